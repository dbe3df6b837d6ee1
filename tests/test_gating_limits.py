"""Gates so far below zero that 1 + exp(-gate) lies near the largest 32-bit number: what comes out is small, not zero."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

GATES = [-80.0, -87.0, -87.5, -88.0, -88.5]


def test_gated_units():
    """silu(g) u in bfloat16 (csrc/rowwise.cu), whose smallest normal number is 2^-126: one rounding of 2^-9, and an exponential of
    2 + 1.16 * 88 units in the last place at most."""
    from tiny_inference_server_b200.kernels import ops
    F = 64
    g = torch.tensor(GATES).to(torch.bfloat16)
    x = torch.empty(len(GATES), 2 * F, dtype=torch.bfloat16)
    x[:, :F], x[:, F:] = g[:, None], 1024.0
    got = ops.swiglu(x.cuda(), torch.empty(len(GATES), F, dtype=torch.bfloat16, device="cuda")).double().cpu()
    want = (g.double() / (1 + torch.exp(-g.double())) * 1024.0)[:, None].expand(-1, F)
    assert float(((got - want) / want).abs().max()) < 2.0 ** -8
    assert float(got.abs().min()) > 0


def test_gate_of_windowed_attention(monkeypatch):
    """One key, so that the values come out as they are, times sigmoid(gate), on the tcgen05 kernel."""
    from tiny_inference_server_b200.kernels import ops
    monkeypatch.setattr(ops, "WINDOW_ATTENTION_TC_MIN_WORK", 0)
    n, H, dim, page = 64, 2, 128, 16
    t = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    pool = torch.full((4, 2, 1, page, dim), 1024.0, dtype=torch.bfloat16, device="cuda")
    pos, slot = t(list(range(n))), t([0] * n)

    class Step:
        positions, row_slot, max_position, decode_only = pos, slot, n - 1, False

        def plan(self, planner):
            return planner.infer(pos, slot)

    gate = torch.tensor([GATES[i % len(GATES)] for i in range(n)]).to(torch.bfloat16)[:, None].expand(-1, H * dim).contiguous()
    out, fault = torch.empty(n, H * dim, dtype=torch.bfloat16, device="cuda"), t([0] * 4)
    before = ops.calls["window_attention_tc"]
    ops.window_attention(torch.zeros(n, H * dim, dtype=torch.bfloat16, device="cuda"), gate.cuda(), out, pool[:, 0], pool[:, 1], t([[0, 1, 2, 3]]),
                         pos, slot, H, page, None, dim ** -0.5, None, None, fault, Step())
    assert ops.calls["window_attention_tc"] == before + 1 and int(fault[0]) == 0
    want = 1024.0 / (1 + torch.exp(-gate.double()))
    got = out.double().cpu()
    assert float(got.abs().min()) > 0
    # (results below 2^-126 have fewer than eight bits)
    assert float((got - want).abs().max()) <= 2.0 ** -134 + float((want * 2.0 ** -8).abs().max())
    assert bool(((got - want).abs() <= want * 2.0 ** -7 + 2.0 ** -133).all()) and math.isfinite(float(got.sum()))
