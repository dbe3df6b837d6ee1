"""Every tile of the tcgen05 product (csrc/gemm_tc.cu): one CTA or a pair of CTAs, 64 to 256 columns, every epilogue, at the edges of
tiles and with several rounds of tiles a CTA."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one row; edges of 128 and 256 rows and of 64 .. 256 columns; a K shorter than a step and one with a remainder; several rounds
@pytest.mark.parametrize("shape", [-1, 0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("M,K,N", [(1, 8, 8), (65, 64, 72), (129, 72, 256), (255, 200, 264), (257, 1536, 192), (300, 520, 200),
                                   (512, 128, 576), (1100, 64, 9000)])
def test_tiles(M, K, N, shape):
    from tiny_inference_server_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K + 8, generator=g, device="cuda").to(torch.bfloat16)[:, 8:]
    w = (torch.randn(K, N + 16, generator=g, device="cuda") * 0.1).to(torch.bfloat16)[:, 16:]
    want = a.double() @ w.double()
    out = torch.full((M, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tc(a, w, out[:, :N], shape=shape)
    scale = a.double().abs() @ w.double().abs()
    # sums of K products in 32 bits, then (bfloat16) one rounding to 8 bits
    bound = scale * (K / 16 + 8) * 2.0 ** -24
    assert bool(((out[:, :N].double() - want).abs() <= bound + want.abs() * 2.0 ** -8).all())
    assert bool((out[:, N:] == 7.0).all())
    if N % 64 == 0:
        gated = torch.full((M, N // 2 + 8), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.gemm_tc(a, w, gated[:, :N // 2], swiglu=True, shape=shape)
        gate, up = want.view(M, -1, 2, 32).unbind(2)
        unit = (torch.nn.functional.silu(gate) * up).reshape(M, -1)
        torch.testing.assert_close(gated[:, :N // 2].double(), unit, rtol=1e-2, atol=1e-3)
        assert bool((gated[:, N // 2:] == 7.0).all())
    assert int(ops.tc_fault()[0]) == 0
