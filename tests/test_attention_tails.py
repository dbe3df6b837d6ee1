"""The last tile of a portion on the tcgen05 attention kernels (csrc/attention_tc.cu, csrc/window_attention_tc.cu): up to 96 of its
128 rows are live, so whole softmax warps have none.  Such a warp leaves the row maxima of its padding rows where the group's
probabilities lie (the first rows of the tile), which the products of the tile before must have read by then: the first
rows of the last tile are compared alone, row by row, and must come out the same every time."""
import pytest
import torch

F64 = torch.float64
TAILS = [(0, 300), (0, 777), (1000, 129), (500, 224), (900, 65)]            # tokens already cached, rows of the portion


def _want(q, k, v, first, scale):
    """The rows of one request at positions first.., all heads, in float64 on the GPU: q (n, H, d), k (m, G, d), v (m, G, e)."""
    n, H, _ = q.shape
    group = H // k.shape[1]
    s = torch.einsum("nhd,mhd->hnm", q.to(F64), k.to(F64).repeat_interleave(group, 1)) * scale
    hidden = torch.arange(k.shape[0], device=q.device)[None] > first + torch.arange(n, device=q.device)[:, None]
    p = torch.softmax(s.masked_fill(hidden, float("-inf")), -1)
    return torch.einsum("hnm,mhe->nhe", p, v.to(F64).repeat_interleave(group, 1))


def _check(got, want, rows):
    """The first eight rows of the last tile: finite, and each as near as bfloat16 probabilities and outputs allow (2^-9 each, at
    random over a row of values; a probability that was overwritten is off by the whole row)."""
    t0 = (rows - 1) // 128 * 128
    got, want = got[t0:t0 + 8].to(F64), want[t0:t0 + 8]
    assert bool(torch.isfinite(got).all())
    off = (got - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
    assert float(off.max()) < 1e-2, off


@pytest.mark.gpu
@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("cached,rows", TAILS)
def test_windowed_attention(cached, rows, shared, monkeypatch):
    from tiny_inference_server_b200.kernels import ops
    monkeypatch.setattr(ops, "WINDOW_ATTENTION_TC_MIN_WORK", 0)
    monkeypatch.setattr(ops, "TC_ATTENTION_MIN_TILES", 1)
    H, G, dim, page = 12, 1 if shared else 3, 128, 16
    gen = torch.Generator(device="cuda").manual_seed(rows)
    bf = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)  # noqa: E731
    m = cached + rows
    pages = -(-m // page)
    table = torch.randperm(pages, generator=gen, device="cuda").to(torch.int32)[None]
    keys = torch.zeros(pages, G, page, dim, dtype=torch.bfloat16, device="cuda")
    values = keys if shared else torch.zeros_like(keys)
    k, v = bf(m, G, dim), bf(m, G, dim)
    at = torch.arange(m, device="cuda")
    keys[table[0, at // page].long(), :, at % page] = k
    if shared:
        v = k
    else:
        values[table[0, at // page].long(), :, at % page] = v
    q = bf(rows, H * dim)
    pos = (cached + torch.arange(rows, device="cuda")).to(torch.int32)
    slot = torch.zeros(rows, dtype=torch.int32, device="cuda")

    class Step:
        positions, row_slot, max_position, decode_only = pos, slot, m - 1, False

        def plan(self, planner):
            return planner.infer(pos, slot)

    fault = torch.zeros(4, dtype=torch.int32, device="cuda")
    want = _want(q.view(rows, H, dim), k, v, cached, dim ** -0.5)
    first = None
    for _ in range(20):
        before = ops.calls["window_attention_tc"]
        out = torch.full((rows, H * dim), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.window_attention(q, None, out, keys, values, table, pos, slot, H, page, None, dim ** -0.5, None, None, fault, Step())
        assert ops.calls["window_attention_tc"] == before + 1
        _check(out.view(rows, H, dim), want, rows)
        assert first is None or torch.equal(out, first)
        first = out
    assert int(fault[0]) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("cached,rows", TAILS)
def test_attention(cached, rows, hd, monkeypatch):
    import kernel_refs as ref
    from tiny_inference_server_b200.kernels import ops
    from tiny_inference_server_b200.kernels.attention_plan import TileSet, plan_tiles
    monkeypatch.setattr(ops, "TC_ATTENTION_MIN_TILES", 1)
    H, KVH, page, m = 12, 3, 16, cached + rows
    gen = torch.Generator().manual_seed(rows)
    bf = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16)  # noqa: E731
    pages = -(-m // page)
    table = torch.randperm(pages, generator=gen).to(torch.int32)[None]
    plane = torch.zeros(pages, 2, KVH, page, hd, dtype=torch.bfloat16)
    k, v = bf(m, KVH, hd), bf(m, KVH, hd)
    for j in range(m):
        plane[table[0, j // page], 0, :, j % page] = ref.cache_row(k[j], j)
        plane[table[0, j // page], 1, :, j % page] = ref.cache_row(v[j], j)
    q = bf(rows, (H + 2 * KVH) * hd)
    t = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    tiles = [([a for a, _ in part], [b for _, b in part]) for part in plan_tiles([(0, rows)], H // KVH)[:3]]
    bound = [(t(a), t(b), len(a)) for a, b in tiles]

    class Step:
        max_position, min_position = m - 1, cached

        def plan(self, planner):
            return TileSet(bound[0], bound[1], max(tiles[0][1], default=0), bound[2], len(tiles[1][0]))

    pos, slot = t(list(range(cached, m))), t([0] * rows)
    want = _want(q[:, :H * hd].cuda().view(rows, H, hd), k.cuda(), v.cuda(), cached, hd ** -0.5)
    q, plane, table, fault = q.cuda(), plane.cuda(), table.cuda(), t([0] * 4)
    first = None
    for _ in range(20):
        before = ops.calls["attn_tc"]
        out = torch.full((rows, H * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(q, out, plane, table, pos, slot, H, KVH, hd, page, None, fault, Step())
        assert ops.calls["attn_tc"] == before + 1
        _check(out.view(rows, H, hd), want, rows)
        assert first is None or torch.equal(out, first)
        first = out
    assert int(fault[0]) == 0
