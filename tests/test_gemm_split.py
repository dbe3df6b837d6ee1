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


# numbers whose parts bfloat16 does not hold, beside numbers so large that the results are ordinary; the same the other way round; results
# that underflow part by part, down to subnormal ones; one step a unit and several rounds of units a CTA, two CTAs a tile
@pytest.mark.parametrize("M,K,N", [(300, 512, 260), (777, 1536, 1536), (520, 32, 9000), (4096, 32, 6144)])
@pytest.mark.parametrize("tiny,huge", [(1e-29, 1e10), (1e-31, 1e12), (1e-36, 1e12), (1e-38, 1e15), (1e-41, 5e34), (1e-41, 1e30), (1e-36, 1.0),
                                       (1e-41, 1.0), (1e-20, 1e-21), (1e-25, 1e-18)])
@pytest.mark.parametrize("swapped", [False, True])
def test_tiny_numbers_meet_huge_ones(M, K, N, tiny, huge, swapped):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(5)
    a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(K, N, generator=g, device="cuda")
    small, large = (w, a) if swapped else (a, w)
    small *= tiny
    large *= huge
    a[7], w[:, 5] = 0.0, 0.0                                    # (zeros stay zeros)
    got, library, want = ops.gemm_split(a, w), torch.mm(a, w), a.double() @ w.double()
    # a multiply-add whose result is subnormal rounds to multiples of 2^-149, K times at most; else as in ordinary products
    assert float((got - want).norm()) <= max(1.05 * float((library - want).norm()), 6e-8 * float(want.norm())) + K * (M * N) ** 0.5 * 2.0 ** -149
    scale = a.double().abs() @ w.double().abs()
    assert bool(((got - want).abs() <= (24 + K) * 2.0 ** -24 * scale + K * 2.0 ** -149).all())
    assert bool((got[7] == 0).all()) and bool((got[:, 5] == 0).all())
    assert int(ops.tc_fault()[0]) == 0


@pytest.mark.parametrize("M,K,N", [(777, 1536, 1536), (4096, 64, 6144)])
def test_some_tiny_numbers_among_ordinary_ones(M, K, N):
    """An infinity changes its own row and nothing else; a few numbers that cannot be split, and a large one that they meet, leave the tiles of
    other rows and columns as they are and their own tile's results as good as multiply-adds."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(6)
    a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(K, N, generator=g, device="cuda") * 0.02
    plain, rows = ops.gemm_split(a, w), torch.arange(M, device="cuda")
    infinite = a.clone()
    infinite[3, 7] = float("inf")
    got = ops.gemm_split(infinite, w)
    assert torch.equal(got[rows != 3], plain[rows != 3]) and not bool(torch.isfinite(got[3]).any())
    a[200], a[200, 9] = 0.0, 1.2345678e-40
    w[9, 300], w[20, 301] = 1e32, 1e-41
    got, want = ops.gemm_split(a, w), a.double() @ w.double()
    assert bool(((got[200] - want[200]).abs() <= want[200].abs() * 2.0 ** -22 + K * 2.0 ** -149).all())
    scale = a.double().abs() @ w.double().abs()
    assert bool(((got - want).abs() <= (24 + K) * 2.0 ** -24 * scale + K * 2.0 ** -149).all())
    assert torch.equal(got[256:, :192], plain[256:, :192]) and torch.equal(got[:, 384:][rows != 200], plain[:, 384:][rows != 200])


def test_products_in_a_graph():
    """Two CTAs a tile add to a result that is set to zero before: inside a graph at every replay, with the inputs of that replay."""
    ops = _ops()
    a, w = torch.randn(777, 1536, device="cuda"), torch.randn(1536, 1536, device="cuda") * 0.02
    ops.gemm(a, w)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    before = ops.calls["gemm_split"]
    with torch.cuda.graph(graph):
        out = ops.gemm(a, w)
    assert ops.calls["gemm_split"] == before + 1
    for seed in range(3):
        a.copy_(torch.randn(777, 1536, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda"))
        graph.replay()
        assert torch.equal(out, ops.gemm_split(a, w)) and _error(out, a.double() @ w.double()) < 1e-6
