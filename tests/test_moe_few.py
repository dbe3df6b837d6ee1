"""Routed experts: few rows with every chosen expert's matrices streamed once (csrc/moe_few.cu) against float64 and beside the
kernels that take a dot product per output element; the router's kernel for many rows against the one for few, bit for bit; the
sum of many rows' choices in vectors against the one in pairs."""
import pytest
import torch

from kernel_refs import gated

pytestmark = pytest.mark.gpu


def _experts(n, d, F, E, top, act=None, weigh=False, shared=False, chosen=None, few=True, seed=0):
    """Error against float64 (2-norm over 2-norm) of moe_experts with the streaming kernels on or off."""
    from tiny_inference_server_b200.kernels import ops
    gen = torch.Generator().manual_seed(seed)
    bf = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(torch.bfloat16)  # noqa: E731
    x, gu = bf(n, d + 8)[:, :d], bf(E, F, d, std=d ** -0.5) if act else bf(E, 2, F, d, std=d ** -0.5)
    down, sh = bf(E, d, F, std=F ** -0.5), bf(n, d) if shared else None
    if chosen is None:
        chosen = torch.stack([torch.randperm(E, generator=gen)[:top] for _ in range(n)])
    w, sg = torch.rand(n, top, generator=gen), torch.rand(n, generator=gen)
    X, GU, D = x.double(), gu.double(), down.double()
    want = torch.zeros(n, d, dtype=torch.float64)
    for r in range(n):
        for k in range(top):
            e = int(chosen[r, k])
            if e < 0:
                continue
            iw = w[r, k].double() if weigh else 1.0
            if act:
                h = torch.relu(GU[e] @ X[r] * iw) ** 2
            else:
                h = gated(GU[e, 0] @ X[r] * iw, GU[e, 1] @ X[r] * iw)
            want[r] += (1.0 if weigh else w[r, k].double()) * (D[e] @ h)
        if shared:
            want[r] += sg[r].double() * sh[r].double()
    c = lambda t: None if t is None else t.cuda()  # noqa: E731
    wide = torch.zeros(n, d + 8, dtype=torch.bfloat16, device="cuda")
    xc = wide[:, :d]
    xc.copy_(x)
    keep, ops.MOE_FEW_MAX_PAIRS = ops.MOE_FEW_MAX_PAIRS, 384 if few else 0
    grouped, ops.MOE_GROUPED_MIN_PAIRS = ops.MOE_GROUPED_MIN_PAIRS, 0
    many, ops.MOE_FEW_MAX_EXPERTS = ops.MOE_FEW_MAX_EXPERTS, 128
    before = ops.calls["moe_few"]
    try:
        got = ops.moe_experts(xc, c(chosen).int(), c(w), c(gu), c(down), c(sh), c(sg) if shared else None, act=act, weigh_input=weigh)
    finally:
        ops.MOE_FEW_MAX_PAIRS, ops.MOE_GROUPED_MIN_PAIRS, ops.MOE_FEW_MAX_EXPERTS = keep, grouped, many
    assert ops.calls["moe_few"] - before == int(few)
    return float((got.double().cpu() - want).norm() / want.norm())


def _check(*args, **options):
    # the hidden elements and the outputs are rounded to bfloat16 (2^-9 each), the sums are 32-bit in both
    few, dots = _experts(*args, few=True, **options), _experts(*args, few=False, **options)
    assert few < 4e-3 and few < 1.1 * dots + 1e-4, (few, dots)


@pytest.mark.parametrize("n,d,F,E,top", [(1, 64, 32, 4, 2), (8, 1536, 1024, 16, 3), (3, 768, 64, 70, 5), (5, 2400, 96, 9, 2), (31, 96, 160, 5, 3), (33, 160, 64, 40, 1), (96, 128, 96, 7, 4)])
@pytest.mark.parametrize("options", [{}, {"act": "relu2"}, {"weigh": True, "shared": True}])
def test_few_rows(n, d, F, E, top, options):
    _check(n, d, F, E, top, **options)


def test_all_rows_on_one_expert_and_choices_of_none():
    _check(70, 64, 64, 6, 2, chosen=torch.tensor([[3, 5]] * 70), shared=True)
    chosen = torch.tensor([[3, 5]] * 9)
    chosen[4] = torch.tensor([-1, 2])
    _check(9, 64, 64, 6, 2, chosen=chosen, shared=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,E,top,groups,keep", [(512, 5, 2, 0, 0), (1536, 16, 3, 4, 2), (2048, 12, 4, 3, 2), (3072, 16, 1, 0, 0), (1024, 17, 9, 0, 0)])
@pytest.mark.parametrize("scores,best,renorm", [("sigmoid", "two_best", True), ("softmax_chosen", "two_best", True), ("softmax", "best", False)])
@pytest.mark.parametrize("correction", [False, True])
@pytest.mark.parametrize("n", [1, 150, 2500])
def test_router_with_its_matrix_in_registers(dtype, d, E, top, groups, keep, scores, best, renorm, correction, n):
    """Bit for bit the kernel that takes a CTA a row, which the same rows reach in a tensor with another row stride."""
    from tiny_inference_server_b200.kernels import ops
    gen = torch.Generator().manual_seed(d + E)
    x = torch.randn(n, d, generator=gen).to(dtype).cuda()
    w = torch.randn(E, d, generator=gen) * d ** -0.5
    w[E // 2] = w[0]                                          # a tie: the lower index wins
    w, sg = w.cuda(), torch.randn(d, generator=gen).cuda()
    corr = (torch.rand(E, generator=gen) * 0.3).cuda() if correction else None
    route = lambda t: ops.moe_route(t, w, corr, sg, groups, keep, top, scores=scores, group_score=best, renorm=renorm)  # noqa: E731
    held = torch.zeros(n, d + 4, dtype=dtype, device="cuda")
    held[:, :d] = x
    for a, b in zip(route(x), route(held[:, :d])):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n,d,F,E,top", [(400, 192, 64, 6, 3), (350, 200, 64, 6, 5), (33, 512, 64, 6, 3), (40, 576, 128, 32, 4)])
def test_many_rows_sorted_and_summed(n, d, F, E, top):
    """Widths of whole vectors and not, choices of four and more a row, through the sorted path; from width 512 with few pairs too."""
    from tiny_inference_server_b200.kernels import ops
    import kernel_refs as ref
    gen = torch.Generator().manual_seed(d)
    bf = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(torch.bfloat16)  # noqa: E731
    x, gu, down, sh = bf(n, d), bf(E, 2, F, d, std=d ** -0.5), bf(E, d, F, std=F ** -0.5), bf(n, d)
    chosen = torch.stack([torch.randperm(E, generator=gen)[:top] for _ in range(n)]).int()
    w, sg = torch.rand(n, top, generator=gen), torch.rand(n, generator=gen)
    want = ref.moe_experts(x, chosen, w, gu, down, sh, sg).double()
    before = ops.calls["moe_grouped_tc"]
    got = ops.moe_experts(x.cuda(), chosen.cuda(), w.cuda(), gu.cuda(), down.cuda(), sh.cuda(), sg.cuda()).double().cpu()
    assert ops.calls["moe_grouped_tc"] - before == int(d % 64 == 0)
    assert float((got - want).norm() / want.norm()) < 8e-3
