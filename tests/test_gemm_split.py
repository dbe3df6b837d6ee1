"""float32 products on the tensor cores (csrc/gemm_split.cu), against 64 bits and beside the library's product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from tiny_inference_server_b200.kernels import ops
    return ops


def _error(got, want):
    return float((got.double() - want).norm() / want.norm())


# edges of tiles (128 rows, 192 columns, 32 of the sum), remainders, one tile and several rounds of tiles, shares of K, a
# sum shorter than a step
@pytest.mark.parametrize("M,K,N", [(1, 4, 4), (65, 32, 192), (128, 36, 196), (129, 200, 188), (300, 1536, 1536), (777, 1536, 640),
                                   (777, 1540, 6144), (2048, 256, 260), (128, 4096, 192)])
def test_split_products_are_no_further_off_than_the_library(M, K, N):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(M, K + 4, generator=g, device="cuda")[:, 4:]
    w = torch.randn(K, N + 8, generator=g, device="cuda")[:, 8:] * 0.02
    want = a.double() @ w.double()
    got = ops.gemm_split(a, w)
    library = torch.mm(a, w)
    # of short sums the library's error is below a last place; of long ones it grows with their length, the split's with their 32nd part
    assert _error(got, want) <= max(1.05 * _error(library, want), 6e-8)
    scale = a.double().abs() @ w.double().abs()
    # per element: 24 roundings toward zero of at most 2^-24 in a step of 32 terms, one rounding to nearest for each step
    bound = (24 + K / 32) * 2.0 ** -24
    assert float(((got.double() - want).abs() / scale).max()) <= bound
    out = torch.full((M, N + 4), 7.0, device="cuda")
    ops.gemm_split(a, w, out[:, :N])
    assert torch.equal(out[:, :N], got) and bool((out[:, N:] == 7.0).all())
    assert int(ops.tc_fault()[0]) == 0


@pytest.mark.parametrize("M,K,N", [(300, 512, 260), (777, 1536, 1536)])
def test_numbers_at_the_limits(M, K, N):
    """Infinities, NaN, the largest numbers and very small ones come out as from multiply-adds."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randn(M, K, generator=g, device="cuda")
    w = torch.randn(K, N, generator=g, device="cuda") * 0.02
    a[3, 7] = float("inf")
    a[5, 1] = float("nan")
    a[9, 0], a[9, 1:] = 3.4028e38, 0.0           # rounds to an infinity in bfloat16
    a[11] *= 1e-33                               # the small parts of these are below what bfloat16 holds
    a[12] = 0.0
    a[130:260] = float("nan")                    # more than a tile of them
    w[2, 100] = float("-inf")
    got, want = ops.gemm_split(a, w), torch.mm(a.double(), w.double())
    library = torch.mm(a, w)
    assert torch.equal(torch.isnan(got), torch.isnan(library))
    inf = torch.isinf(library)
    assert torch.equal(got[inf], library[inf]) and torch.equal(torch.isinf(got), inf)
    assert bool((got[12][library[12] == 0] == 0).all())
    keep = torch.ones(M, dtype=torch.bool, device="cuda")
    keep[[3, 5]] = False
    keep[130:260] = False
    cols = torch.arange(N, device="cuda") != 100
    for r in (9, 11):
        assert _error(got[r][cols], want[r][cols]) < 2e-6
    assert _error(got[keep][:, cols], want[keep][:, cols]) < 2e-6


def test_products_go_where_their_operands_allow():
    ops = _ops()
    a, w = torch.randn(800, 1024, device="cuda"), torch.randn(1024, 512, device="cuda")
    many = torch.randn(1024, 8192, device="cuda")
    for x, y, kernel in ((a, w, True), (a[:ops.SPLIT_MIN_ROWS], many, True), (a[:ops.SPLIT_MIN_ROWS - 1], many, False), (a, w[:, :256], False),
                         (a[:, :512], w[:512], False), (a[:, 1:], w[1:], False), (a[:, :1023], w[:1023], False),
                         (a, w.t().contiguous().t(), False), (a, w[:, :510], False), (a, w[:, 1:509], False), (a, w[:, 4:508], True)):
        before = ops.calls["gemm_split"]
        got = ops.gemm(x, y)
        assert (ops.calls["gemm_split"] > before) == kernel
        assert _error(got, x.double() @ y.double()) < 1e-6
