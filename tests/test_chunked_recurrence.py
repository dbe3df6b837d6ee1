"""The chunked form of the matrix-state recurrences (csrc/chunked_recurrence.cu) against the recurrence walked in float64,
beside the kernels that walk it token by token: every kind of decay, both widths, portions around the edges of a chunk (64
tokens) and of its sub-chunks (16), several requests of unequal length with a state of their own, strided rows, decays that
underflow, and non-finite tokens, which no earlier token may see."""
import math

import pytest
import torch

F64 = torch.float64


def _walk(q, k, v, g, S, beta=None, bonus=None):
    """o_t = S_t^T q_t over the tokens in float64; ``beta``: the delta rule; ``bonus``: outputs read the state before."""
    out = []
    for t in range(len(q)):
        if bonus is not None:
            out.append(torch.einsum("hdv,hd->hv", S, q[t]) + (bonus * q[t] * k[t]).sum(-1, keepdim=True) * v[t])
        S = g[t][..., None] * S
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][..., None] * u[:, None]
        if bonus is None:
            out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    return torch.stack(out), S


def _norm(o, w, eps):
    return o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps) * w


class Case:
    """Inputs of a step in ``dtype`` and its oracle; ``call(ops, segments)`` runs one of the entry points."""

    def __init__(self, rule, K, V, lengths, dtype, seed=0, H=4, strong=0.0):
        self.rule, self.K, self.V, self.lengths, self.dtype, self.H = rule, K, V, list(lengths), dtype, H
        gen = torch.Generator().manual_seed(seed)
        n = sum(lengths)
        r = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
        self.G = G = 2 if rule in ("channel", "head", "step") else H
        self.n, self.eps = n, 1e-6
        cols = (G if rule == "forget" else 2 * G) * K + H * V + (H * V if rule == "bonus" else 0)
        self.rows = r(n, cols + 16).to(dtype)[:, :cols]                          # a view with a longer row
        self.a = (r(n, H if rule in ("head", "step") else H * K) + strong).to(dtype)
        self.b, self.gate = r(n, H).to(dtype), r(n, H * V).to(dtype)
        self.a_log = {"constant": 1 - 2.0 ** -(2 + torch.arange(H).float()), "gated": torch.full((H,), 0.125),
                      "forget": torch.rand(H * K, generator=gen) * 0.9, "bonus": r(H * K)}.get(rule, r(H) * 0.3)
        self.bias = torch.rand(H if rule in ("head", "step") else H * K, generator=gen) * 3 - 2
        self.norm_w = 1 + 0.1 * r(H * V if rule in ("constant", "bonus") else V)
        slots = len(lengths)
        self.state = r(slots + 1, H * K * V + 8)[:, :H * K * V] * 0.1            # a free stride between the slots
        order = list(range(slots))[::-1]                                         # requests in slots of another order
        self.slot = torch.cat([torch.full((m,), order[i], dtype=torch.int32) for i, m in enumerate(lengths)])
        ends = torch.tensor(lengths).cumsum(0)
        self.last = torch.cat([torch.full((m,), int(e) - 1, dtype=torch.int32) for m, e in zip(lengths, ends)])
        self.first = [int(e) - m for m, e in zip(lengths, ends)]
        self.order = order

    def oracle(self):
        H, G, K, V, rule = self.H, self.G, self.K, self.V, self.rule
        d = self.rows.to(F64)
        a, bias, a_log, gate = self.a.to(F64), self.bias.to(F64), self.a_log.to(F64), self.gate.to(F64)
        silu, plus = torch.nn.functional.silu, torch.nn.functional.softplus
        out, states = torch.zeros(self.n, H * V, dtype=F64), self.state.to(F64).clone()
        for r0, m, s in zip(self.first, self.lengths, self.order):
            x, ar = d[r0:r0 + m], a[r0:r0 + m]
            S, beta, bonus = states[s].view(H, K, V), None, None
            vec = lambda at, w, heads: x[:, at:at + heads * w].reshape(m, heads, w)  # noqa: E731
            q = vec(0, K, G)
            if rule == "forget":
                v = vec(G * K, V, H)
                low = a_log.view(H, K)
                g = low + (1 - low) * torch.sigmoid(ar.view(m, H, K) + bias.view(H, K))
                q, k = silu(q), 1 - g
            else:
                k, v = vec(G * K, K, G), vec(2 * G * K, V, H)
                if rule in ("channel", "head"):
                    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
                    q, beta = q * K ** -0.5, torch.sigmoid(self.b[r0:r0 + m].to(F64))
                    z = (ar + bias).view(m, H, -1)
                    g = torch.exp(-torch.exp(a_log)[:, None] * plus(z)).expand(m, H, K)
                elif rule == "constant":
                    q, k, v, g = silu(q), silu(k), silu(v), a_log[:, None].expand(m, H, K)
                elif rule == "gated":
                    q, g = q * K ** -0.5, torch.exp(-plus(-(ar + bias)).view(m, H, K) * a_log[:, None])
                elif rule == "step":
                    dt = plus(ar + bias)
                    g, v = torch.exp(-torch.exp(a_log) * dt)[..., None].expand(m, H, K), v * dt[..., None]
                else:
                    g, bonus = torch.exp(-torch.exp((ar + bias).view(m, H, K))), a_log.view(H, K)
            q, k = (t.repeat_interleave(H // t.shape[1], 1) for t in (q, k))
            o, S = _walk(q, k, v, g, S, beta, bonus)
            states[s] = S.reshape(-1)
            gr = gate[r0:r0 + m]
            if rule == "constant":
                y = _norm(o.flatten(1), self.norm_w.to(F64), self.eps) * torch.sigmoid(gr)
            elif rule == "step":
                y = o.flatten(1)
            elif rule == "bonus":
                y = _norm(o, self.norm_w.to(F64).view(H, V), self.eps).flatten(1) * silu(x[:, -H * V:])
            else:
                y = _norm(o, self.norm_w.to(F64), self.eps).flatten(1)
                y = y if rule == "forget" else y * (silu(gr) if rule == "gated" else torch.sigmoid(gr))
            out[r0:r0 + m] = y
        return out, states

    def call(self, ops, segments, rows_at=0, state_at=0):
        """``rows_at``, ``state_at``: elements that the rows and the states begin beside a boundary."""
        c = lambda t: t.cuda()  # noqa: E731
        wide = torch.empty(self.n, self.rows.shape[1] + 16, dtype=self.dtype, device="cuda")
        rows = wide[:, rows_at:rows_at + self.rows.shape[1]]
        rows.copy_(self.rows)
        held = torch.empty(self.state.shape[0], self.state.shape[1] + 8, device="cuda")
        state = held[:, state_at:state_at + self.state.shape[1]]
        state.copy_(self.state)
        out = torch.zeros(self.n, self.H * self.V, dtype=self.dtype, device="cuda")
        tail = dict(requests=len(self.lengths), segments=segments)
        at = (c(self.slot), c(self.last), self.H)
        if self.rule in ("channel", "head"):
            ops.delta_rule(rows, c(self.b), c(self.a), c(self.gate), c(self.a_log), c(self.bias), c(self.norm_w), self.eps, 1e-6,
                           self.K ** -0.5, state, out, *at, self.G, self.K, self.V, decay_per_head=self.rule == "head", **tail)
        elif self.rule == "constant":
            ops.linear_attention(rows, c(self.gate), c(self.a_log), c(self.norm_w), self.eps, state, out, *at, self.K, self.V, **tail)
        elif self.rule == "forget":
            ops.forget_gate_recurrence(rows, c(self.a), c(self.a_log), c(self.bias), c(self.norm_w), self.eps, state, out, *at,
                                       self.K, self.V, **tail)
        elif self.rule == "gated":
            ops.gated_linear_attention(rows, c(self.a), c(self.a_log), c(self.bias), c(self.gate), c(self.norm_w), self.eps,
                                       self.K ** -0.5, state, out, *at, self.K, self.V, **tail)
        elif self.rule == "step":
            out = ops.state_space_scan(rows, c(self.a), c(self.a_log), c(self.bias), state, *at, self.G, self.K, self.V, **tail)
        else:
            ops.time_mix(rows, c(self.a), c(self.a_log), c(self.bias), c(self.norm_w), self.eps, state, out, *at, self.K, **tail)
        return out.double().cpu(), state.double().cpu()

    def segments(self, chunked):
        return torch.tensor(self.first, dtype=torch.int32, device="cuda"), len(self.first), 10 ** 6 if chunked else 1


def _off(got, want):
    return float((got - want).norm() / want.norm())


RULES = ["channel", "head", "constant", "forget", "gated", "step", "bonus"]


def _compare(case):
    from tiny_inference_server_b200.kernels import ops
    want_o, want_s = case.oracle()
    walked_o, walked_s = case.call(ops, case.segments(False))
    before = ops.calls["recurrence_chunked"]
    got_o, got_s = case.call(ops, case.segments(True))
    assert ops.calls["recurrence_chunked"] == before + 1
    # 32-bit sums of at most K + 64 products a chunk, errors of one chunk carried on by decays <= 1: a few times 2^-23
    # relative to the whole; and never much worse than the walk, whose chain is as long as the portion
    limit = 3e-6 if case.dtype == torch.float32 or case.rule == "step" else 4e-3
    assert _off(got_o, want_o) < limit, (_off(got_o, want_o), _off(walked_o, want_o))
    assert _off(got_s, want_s) < 3e-6, (_off(got_s, want_s), _off(walked_s, want_s))
    assert _off(got_s, want_s) < 2 * _off(walked_s, want_s) + 3e-7
    assert torch.equal(got_s[-1], case.state[-1].double())                  # nobody's slot


@pytest.mark.gpu
@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K,V,lengths", [(128, 128, (130, 1, 63)), (64, 128, (65,)), (128, 64, (16, 64, 17)), (64, 64, (15, 129))])
def test_chunks_against_the_walk(rule, dtype, K, V, lengths):
    if rule == "bonus" and K != V:
        V = K
    _compare(Case(rule, K, V, lengths, dtype))


@pytest.mark.gpu
@pytest.mark.parametrize("rule", ["channel", "head", "gated", "bonus", "step"])
def test_decays_that_underflow(rule):
    """Decays far below the smallest float beside ones near 1: products are zero, never a division by them."""
    case = Case(rule, 64, 64, (100, 70), torch.float32, seed=3, strong=0.0)
    case.a[::7] += -120.0 if rule == "gated" else 120.0
    case.a[3::7] += 40.0 if rule == "gated" else -40.0
    if rule == "gated":
        case.a_log.fill_(1.0)
    _compare(case)


@pytest.mark.gpu
@pytest.mark.parametrize("rule", RULES)
def test_a_token_that_is_not_finite_shows_in_no_earlier_one(rule):
    from tiny_inference_server_b200.kernels import ops
    case = Case(rule, 64, 64, (90, 40), torch.float32, seed=5)
    clean, _ = case.call(ops, case.segments(True))
    for bad, row in ((math.inf, 37), (math.nan, 70)):
        broken = Case(rule, 64, 64, (90, 40), torch.float32, seed=5)
        broken.rows[row] = bad
        got, states = broken.call(ops, broken.segments(True))
        # the block of 16 tokens around a broken one is summed another way: 32-bit sums of up to 128 products, not the same bits
        assert _off(got[:row], clean[:row]) < 3e-6 and torch.equal(got[90:], clean[90:])
        assert not torch.isfinite(states[broken.order[0]]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_no_further_off_than_the_walk(rule, dtype):
    """States and 32-bit outputs, whatever the activations, in the mean over shapes.  Both forms are off by single roundings
    (2^-24), so a shape's ratio scatters by about 0.1 around 0.5 to 1.05: the mean of five by half of that."""
    from tiny_inference_server_b200.kernels import ops
    out, state = [], []
    for K, V, lengths in ((128, 128, (777,)), (64, 64, (500, 130)), (128, 64, (300,)), (64, 128, (1100,)), (128, 128, (128, 200))):
        case = Case(rule, K, K if rule == "bonus" else V, lengths, dtype, seed=7)
        want_o, want_s = case.oracle()
        walked_o, walked_s = case.call(ops, case.segments(False))
        got_o, got_s = case.call(ops, case.segments(True))
        out.append(_off(got_o, want_o) / _off(walked_o, want_o))
        state.append(_off(got_s, want_s) / _off(walked_s, want_s))
    assert sum(state) / 5 < 1.15, state
    assert sum(out) / 5 < 1.05, out


@pytest.mark.gpu
@pytest.mark.parametrize("rule", RULES)
def test_operands_that_the_chunks_do_not_take_are_walked(rule):
    """A state or rows that start beside a 16-byte boundary, and widths without the kernels: token by token, counted as that."""
    from tiny_inference_server_b200.kernels import ops
    for K, V, rows_at, state_at in ((64, 64, 1, 0), (64, 64, 0, 1), (32, 32, 0, 0)):
        if rule == "bonus" and rows_at:
            continue                                                        # (its walk reads rows in 16-byte vectors as well)
        case = Case(rule, K, V, (70, 9), torch.float32, seed=9)
        want_o, want_s = case.oracle()
        before, launched = ops.calls["recurrence_chunked"], ops.launches
        got_o, got_s = case.call(ops, case.segments(True), rows_at, state_at)
        assert ops.calls["recurrence_chunked"] == before
        assert ops.launches - launched == (1 if rule == "step" else 2)
        assert _off(got_o, want_o) < 3e-6 and _off(got_s, want_s) < 3e-6


def _same_where_not_finite(got, walked):
    """Infinities and NaN where the walk has them, and the same ones; elsewhere 32-bit sums of up to 128 products."""
    assert torch.equal(torch.isnan(got), torch.isnan(walked))
    inf = torch.isinf(walked)
    assert torch.equal(got[inf], walked[inf]) and torch.equal(torch.isinf(got), inf)
    fine = torch.isfinite(walked)
    assert _off(got[fine], walked[fine]) < 3e-6


@pytest.mark.gpu
@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("where", ["value", "key", "query", "decay", "state", "overflow"])
def test_numbers_that_are_not_finite_are_what_the_walk_makes_of_them(rule, where):
    from tiny_inference_server_b200.kernels import ops
    if (where, rule) == ("overflow", "forget"):
        pytest.skip("keys below 1: sums that end near the largest number, and how a sum is grouped decides whether it passes it")
    case = Case(rule, 64, 64, (200, 40, 129), torch.float32, seed=11)
    G, K, H, V = case.G, 64, case.H, 64
    at = {"query": 3, "key": G * K + 3, "value": (G if rule == "forget" else 2 * G) * K + 2 * V + 5}
    if where == "state":
        case.state[case.order[0], 2 * K * V + 7 * V + 9] = math.inf
    elif where == "decay":
        case.a[77, case.a.shape[1] - 1] = math.nan
    elif where == "overflow":                                               # each finite, their sums not
        case.rows[60:90, at["value"]] = 3e38
        case.rows[60:90, at["key"]:at["key"] + 40] = 30.0
    else:
        case.rows[100, at[where]] = math.inf
        case.rows[240 + 100, at[where] + 1] = -math.inf
    walked = case.call(ops, case.segments(False))
    before = ops.calls["recurrence_chunked"]
    got = case.call(ops, case.segments(True))
    assert ops.calls["recurrence_chunked"] == before + 1
    for g, w in zip(got, walked):
        _same_where_not_finite(g, w)


def test_who_is_taken_in_chunks():
    """The requests of a step, the longest first; only portions that may be long enter the chunks, from a length that depends
    on the rule, or from a shorter one where there are several."""
    from tiny_inference_server_b200.kernels import ops, segment_plan
    planner = segment_plan.planner()

    def portions(decay, lengths):
        first = [sum(lengths[:i]) for i in range(len(lengths))]
        arrays, facts = planner.plan(list(zip(first, lengths)))
        seg = planner.bind({k: torch.tensor(v) for k, v in arrays.items()}, facts)
        assert seg.count == len(lengths) == len(seg.row0) and seg.longest == max(lengths)
        ordered = [lengths[first.index(int(r))] for r in seg.row0]
        assert sorted(ordered) == sorted(lengths) and ordered == sorted(lengths, reverse=True)
        assert list(seg.rows) == [m for m in ordered if m >= segment_plan.LISTED_ROWS]
        return ops._chunk_portions(decay, seg, sum(lengths))

    assert portions("channel", [159]) == (0, 0) and portions("channel", [160]) == (1, 160)
    assert portions("channel", [1] * 31 + [239]) == (0, 0) and portions("channel", [1] * 31 + [240]) == (1, 240)
    assert portions("channel", [20] * 20 + [224]) == (0, 0) and portions("channel", [1] * 7 + [224]) == (1, 224)
    assert portions("bonus", [1] * 31 + [511]) == (0, 0) and portions("bonus", [1] * 31 + [512]) == (1, 512)
    assert portions("gated", [1, 300, 1, 47, 48, 700]) == (3, 1048)
    assert portions("channel", [128] * 4) == (4, 512) and portions("channel", [64] * 16 + [224]) == (17, 1248)
    assert portions("channel", [64] * 16) == (0, 0)                          # none of them long
    assert portions("bonus", [128] * 8) == (0, 0) and portions("bonus", [192] * 8) == (8, 1536)
    assert portions("step", [1] * 8) == (0, 0)
    arrays, facts = planner.plan_decode(5)
    assert ops._chunk_portions("step", planner.bind({k: torch.tensor(v) for k, v in arrays.items()}, facts), 5) == (0, 0)
    assert ops._chunk_portions("step", None, 5) == (0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("lengths", [(1, 1, 200, 5, 530, 1), (530,) + (1,) * 40, (40, 600, 48)])
def test_a_step_with_single_rows_beside_long_portions(rule, lengths):
    """Long portions in chunks, the other requests token by token, both against the recurrence in float64."""
    from tiny_inference_server_b200.kernels import ops, segment_plan
    case = Case(rule, 64, 64, lengths, torch.float32, seed=13)
    want_o, want_s = case.oracle()
    planner = segment_plan.planner()
    arrays, facts = planner.plan(list(zip(case.first, case.lengths)))
    seg = planner.bind({k: torch.tensor(v, dtype=torch.int32, device="cuda") for k, v in arrays.items()}, facts)
    before, launched = ops.calls["recurrence_chunked"], ops.launches
    got_o, got_s = case.call(ops, seg)
    assert ops.calls["recurrence_chunked"] == before + 1
    assert ops.launches - launched == (5 if rule == "step" else 6)
    assert _off(got_o, want_o) < 3e-6 and _off(got_s, want_s) < 3e-6
    for r0, m in zip(case.first, case.lengths):                              # every request for itself
        assert _off(got_o[r0:r0 + m], want_o[r0:r0 + m]) < 6e-6


@pytest.mark.gpu
def test_without_memory_for_the_scratch_the_step_is_walked(monkeypatch):
    from tiny_inference_server_b200.kernels import ops
    case = Case("gated", 64, 64, (300, 2), torch.float32, seed=15)
    walked_o, walked_s = case.call(ops, case.segments(False))
    empty = torch.empty

    def full(*size, **options):
        if len(size) == 1 and isinstance(size[0], int) and size[0] > 100000:
            raise torch.cuda.OutOfMemoryError("no memory left")
        return empty(*size, **options)

    segments, before = case.segments(True), ops.calls["recurrence_chunked"]
    monkeypatch.setattr(torch, "empty", full)
    got_o, got_s = case.call(ops, segments)
    assert ops.calls["recurrence_chunked"] == before
    assert torch.equal(got_o, walked_o) and torch.equal(got_s, walked_s)
