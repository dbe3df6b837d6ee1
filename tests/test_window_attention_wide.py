"""Windowed attention on the kernels that read whole pages by TMA boxes, against the formula in float64 and beside the mma.sync
kernel: long portions on the tcgen05 kernel (csrc/window_attention_tc.cu): widths, shared value rows, windows and chunks, biases
(also ones that vary by more than the first pass's slack within a tile), sinks, bounds, both gates, portions around the edges of
a tile of 128 rows behind cached keys, page sizes, requests side by side with single rows, and pages whose unseen rows are not
finite; the rows of decode steps on the kernel whose key shares are a cluster (csrc/window_attention_decode.cu), likewise."""
import math

import pytest
import torch

F64 = torch.float64


@pytest.fixture(autouse=True)
def steps_of_any_size(monkeypatch):
    """The tcgen05 kernel also where a step's work is too small for it to pay."""
    from tiny_inference_server_b200.kernels import ops
    monkeypatch.setattr(ops, "WINDOW_ATTENTION_TC_MIN_WORK", 0)
    monkeypatch.setattr(ops, "WINDOW_ATTENTION_TC_MIXED_ROWS", 0)


class _Step:
    def __init__(self, pos, slot, decode_only):
        self.positions, self.row_slot, self.max_position, self.decode_only = pos, slot, int(pos.max()), decode_only

    def plan(self, planner):
        return planner.infer(self.positions, self.row_slot)


def _oracle(q, k, v, first, scale, window, r1, r2, sink, cap):
    """q (n, H, d) at positions first.., k (m, G, d), v (m, G, e)."""
    n, H, _ = q.shape
    group = H // k.shape[1]
    pos, key = torch.arange(first, first + n), torch.arange(k.shape[0])
    dist = pos[:, None] - key[None]
    low = torch.zeros_like(pos) if not window else ((pos - window + 1).clamp(min=0) if window > 0 else pos - pos % -window)
    hidden = (dist < 0) | (key[None] < low[:, None])
    out = torch.empty(n, H, v.shape[2], dtype=F64)
    for h in range(H):
        s = q[:, h] @ k[:, h // group].t() * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if r1 is not None:
            s = s - r1[h] * torch.log1p(r2[h] * dist.clamp(min=0))
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :k.shape[0]] @ v[:, h // group]
    return out


def _run(name, K, V, H, G, portions, page, window=0, bias=None, sink=False, cap=None, gate=None, shared=False, seed=0):
    """``portions``: [(tokens already cached, rows of the step)].  ``name``: the kernel, ``tc`` or ``decode``.  Returns (its error,
    that of the mma.sync kernel), 2-norm over 2-norm against float64."""
    from tiny_inference_server_b200.kernels import ops
    gen = torch.Generator().manual_seed(seed)
    bf = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16)  # noqa: E731
    n = sum(r for _, r in portions)
    pages_of = [-(-(h + r) // page) for h, r in portions]
    total = sum(pages_of) + 3
    # rows that nobody wrote hold what another request left: not finite
    width = K if shared else K + V
    pool = torch.full((total, G * page * width), math.nan, dtype=torch.bfloat16)
    kp = pool[:, :G * page * K].view(total, G, page, K)
    vp = kp[..., :V] if shared else pool[:, G * page * K:].view(total, G, page, V)
    perm = torch.randperm(total, generator=gen).to(torch.int32)
    table = torch.full((len(portions), max(pages_of) + 2), -1, dtype=torch.int32)
    q, scale = bf(n, H * K), K ** -0.5
    r1 = r2 = None
    if bias is not None:
        r1, r2 = bias * (0.2 + torch.rand(H, generator=gen)), 0.1 + 2 * torch.rand(H, generator=gen)
    snk = torch.randn(H, generator=gen) * 2 if sink else None
    g = {None: None, "head": bf(n, H), "element": bf(n, H * V)}[gate]
    want, at, used = [], 0, 0
    pos, slot = [], []
    for i, (h, r) in enumerate(portions):
        ids = perm[used:used + pages_of[i]]
        used += pages_of[i]
        first_page = 0 if not window else max(0, (h - window + 1 if window > 0 else h - h % -window)) // page
        table[i, first_page:pages_of[i]] = ids[first_page:]                 # pages behind the window have been given back
        k, v = bf(h + r, G, K), bf(h + r, G, V)
        if shared:
            v = k[..., :V]
        for j in range(h + r):
            kp[ids[j // page], :, j % page] = k[j]
            if not shared:
                vp[ids[j // page], :, j % page] = v[j]
        o = _oracle(q[at:at + r].double().view(r, H, K), k.double(), v.double(), h, scale, window,
                    None if r1 is None else r1.double(), None if r2 is None else r2.double(), None if snk is None else snk.double(), cap)
        if gate == "head":
            o = o * torch.sigmoid(g[at:at + r].double())[..., None]
        elif gate == "element":
            o = o * torch.sigmoid(g[at:at + r].double()).view(r, H, V)
        want.append(o.flatten(1))
        pos += list(range(h, h + r))
        slot += [i] * r
        at += r
    want = torch.cat(want)
    c = lambda t: None if t is None else t.cuda()  # noqa: E731
    dev = pool.cuda()
    dk = dev[:, :G * page * K].view(total, G, page, K)
    dv = dk[..., :V] if shared else dev[:, G * page * K:].view(total, G, page, V)
    pos, slot = torch.tensor(pos, dtype=torch.int32, device="cuda"), torch.tensor(slot, dtype=torch.int32, device="cuda")
    off = []
    for on in (True, False):
        switch = f"WINDOW_ATTENTION_{name.upper()}"
        keep = getattr(ops, switch)
        setattr(ops, switch, on)
        fault = torch.zeros(4, dtype=torch.int32, device="cuda")
        out = torch.full((n, H * V), 7.0, dtype=torch.bfloat16, device="cuda")
        before = ops.calls[f"window_attention_{name}"]
        try:
            ops.window_attention(c(q), c(g), out, dk, dv, c(table), pos, slot, H, page, abs(window) or None, scale, c(r1), c(r2),
                                 fault, _Step(pos, slot, name == "decode"), sink=c(snk), gate_per_head=gate == "head",
                                 chunked=window < 0, softcap=cap)
        finally:
            setattr(ops, switch, keep)
        assert ops.calls[f"window_attention_{name}"] - before == int(on)
        assert int(fault[0]) == 0
        off.append(float((out.double().cpu() - want).norm() / want.norm()))
    return off


def _check(off):
    # probabilities and outputs rounded to bfloat16 (2^-9 each, at random), both kernels alike
    assert off[0] < 5e-3 and off[0] < 1.1 * off[1] + 2e-4, off


@pytest.mark.gpu
@pytest.mark.parametrize("K,shared,options", [(128, False, {"window": 1024, "bias": 0.5, "gate": "element"}), (128, False, {"bias": 4.0}),
                                              (128, False, {"sink": True}), (192, True, {}), (128, False, {})])
def test_no_further_off_than_the_mma_kernel(K, shared, options):
    """The mean over three seeds of the error over the mma.sync kernel's, which scatters by 0.003: both round the probabilities to
    bfloat16 relative to the row's maximum."""
    off = [_run("tc", K, 128, 4, 1, [(0, 500), (200, 300)], 16, shared=shared, seed=s, **options) for s in range(3)]
    assert sum(a / b for a, b in off) / 3 < 1.01, off


@pytest.mark.gpu
@pytest.mark.parametrize("K,V,shared", [(128, 128, False), (192, 128, True), (128, 128, True), (64, 128, False), (128, 64, False),
                                        (64, 64, False)])
@pytest.mark.parametrize("portions", [[(0, 300)], [(77, 129), (0, 64), (500, 1)], [(1000, 128), (3, 127)]])
def test_widths_and_portions(K, V, shared, portions):
    _check(_run("tc", K, V, 4, 1 if shared else 2, portions, 16, shared=shared))


@pytest.mark.gpu
@pytest.mark.parametrize("page", [16, 32, 128])
@pytest.mark.parametrize("window", [0, 1, 100, 128, 300, -64, -200])
def test_windows_and_pages(page, window):
    _check(_run("tc", 128, 128, 2, 1, [(190, 257), (0, 65)], page, window=window, gate="element"))


@pytest.mark.gpu
@pytest.mark.parametrize("bias", [0.5, 4.0, 60.0, -0.7])
@pytest.mark.parametrize("window", [0, 200])
def test_biases(bias, window):
    _check(_run("tc", 128, 128, 4, 2, [(300, 260), (0, 90)], 16, window=window, bias=bias, gate="element"))


@pytest.mark.gpu
@pytest.mark.parametrize("options", [{"sink": True}, {"cap": 3.0}, {"cap": 3.0, "window": -128, "sink": True}, {"gate": "head", "sink": True}])
@pytest.mark.parametrize("K,shared", [(128, False), (192, True)])
def test_sinks_bounds_and_gates(options, K, shared):
    _check(_run("tc", K, 128, 4, 1, [(130, 200), (0, 70)], 16, shared=shared, **options))


# single rows: one key, the edges of a tile of 64 keys, few and many shares of the keys
ROWS = [[(0, 1), (63, 1), (64, 1), (65, 1), (700, 1)], [(2500, 1)], [(h * 37 % 400, 1) for h in range(40)]]


@pytest.mark.gpu
@pytest.mark.parametrize("K,V,H,G,shared", [(128, 128, 12, 3, False), (192, 128, 12, 1, True), (128, 128, 16, 1, True), (64, 128, 4, 2, False),
                                            (128, 64, 6, 2, False), (256, 128, 4, 4, False), (64, 64, 2, 2, False)])
@pytest.mark.parametrize("portions", ROWS)
def test_single_rows(K, V, H, G, shared, portions):
    _check(_run("decode", K, V, H, G, portions, 16, shared=shared))


@pytest.mark.gpu
@pytest.mark.parametrize("options", [{"sink": True}, {"cap": 3.0}, {"gate": "head", "sink": True}, {"gate": "element", "bias": 0.5},
                                     {"bias": 30.0}, {"cap": 3.0, "window": -128, "sink": True}, {"window": 1}, {"window": 100},
                                     {"window": 64, "bias": 0.5}])
@pytest.mark.parametrize("page", [16, 64, 128])
def test_single_rows_with_all_they_may_ask_for(options, page):
    _check(_run("decode", 128, 128, 8, 2, ROWS[0] + [(1500, 1)], page, **options))


def test_tiles_cover_the_rows_once():
    from tiny_inference_server_b200.kernels import window_plan
    for group in (1, 3, 4, 12, 64):
        planner = window_plan.WindowTilePlanner(max(1, window_plan.PACKED_ROWS // group))
        segments = [(0, 1), (1, 200), (201, 63), (264, 64), (328, 129)]
        arrays, facts = planner.plan(segments)
        tiles = planner.bind({k: torch.tensor(v) for k, v in arrays.items()}, facts)
        rows = lambda t: sorted(r for a, m in zip(t[0].tolist(), t[1].tolist()) for r in range(a, a + m))  # noqa: E731
        assert rows(tiles.rows) == list(range(457)) and len(tiles.rows[0]) == tiles.rows[2]
        wide = list(range(1, 201)) + list(range(264, 457))
        assert rows(tiles.wide) == wide
        covered = tiles.rows_in_wide
        assert rows((tiles.rows[0][:covered], tiles.rows[1][:covered])) == wide
        assert sum(len(v) for v in arrays.values()) <= planner.max_words(457)


def test_shares_of_a_row_keep_all_clusters_resident():
    from tiny_inference_server_b200.kernels import ops
    # as a device answers whose clusters of 16 do not fill it: two CTAs an SM, and one
    two = {(0, 1): 296, (0, 2): 148, (0, 4): 71, (0, 8): 33, (0, 16): 14}
    one = {(0, 1): 148, (0, 2): 74, (0, 4): 33, (0, 8): 15, (0, 16): 7}
    shares = ops._decode_shares
    assert shares(two, 0, 14, 4096, 128, 8) == 16 and shares(two, 0, 15, 4096, 128, 8) == 8
    assert shares(two, 0, 16, 1000, 128, 4) == 8 and shares(two, 0, 400, 4096, 128, 4) == 1
    assert shares(one, 0, 32, 8000, 256, 2) == 4 and shares(one, 0, 8, 1000, 256, 2) == 8
    assert shares(two, 0, 1, 63, 128, 4) == 1 and shares(two, 0, 1, 64, 128, 4) == 2                # a tile of keys each
    # few rows, many keys: more shares than a cluster has
    assert shares(two, 0, 1, 8000, 192, 16) == 16 and shares(two, 0, 1, 16000, 192, 16) == 0
    assert shares(two, 0, 3, 64000, 128, 8) == 16 and shares(one, 0, 16, 16000, 256, 2) == 0
    assert shares(one, 0, 256, 100, 256, 2) == 0 and shares(one, 0, 64, 100, 256, 2) == 2


def test_when_long_portions_are_worth_a_launch(monkeypatch):
    from tiny_inference_server_b200.kernels import ops
    monkeypatch.undo()
    assert ops._wide_tiles_pay(2048, 0, 1024, 12) and not ops._wide_tiles_pay(1200, 0, 1024, 12)
    # beside other tiles, in which one launch runs as long as the rows alone, only portions that take as long themselves
    assert not ops._wide_tiles_pay(1024 + 8, 8, 4000, 12) and not ops._wide_tiles_pay(31 + 512, 31, 4000, 12)
    assert ops._wide_tiles_pay(3072 + 8, 8, 4000, 12)
