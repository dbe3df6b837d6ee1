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


def _gated(a, w, block):
    """silu(gate) * up in 64 bits, gate and up columns in alternating blocks."""
    gate, up = (a.double() @ w.double()).view(a.shape[0], -1, 2, block).unbind(2)
    return (torch.nn.functional.silu(gate) * up).reshape(a.shape[0], -1)


# the first rows that go there; one full tile of 256 and one row more; nine tenths of two, three and four tiles; full tiles
@pytest.mark.parametrize("rows,fused", [(64, False), (65, True), (256, True), (257, False), (460, False), (461, True), (512, True), (513, False),
                                        (691, False), (692, True), (768, True), (921, False), (922, True)])
def test_which_way_gate_and_up_go(rows, fused):
    from tiny_inference_server_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    K, H = 256, 128
    wide = torch.randn(rows, K + 8, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(K, 2 * H, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    for a, block, taken in ((wide[:, 8:], 32, fused), (wide[:, 8:], 64, False), (wide[:, 4:K + 4], 32, False)):   # (the last: 8 bytes behind a boundary)
        before = ops.calls["gemm_tc"]
        got = ops.gemm_swiglu(a, w, H, block)
        assert ops.calls["gemm_tc"] == before + taken
        torch.testing.assert_close(got.double(), _gated(a, w, block), rtol=2e-2, atol=2e-3)
