"""Every page size of the tcgen05 attention kernel (csrc/attention_tc.cu), whose boxes two warps order in turns: 16 boxes a key tile
(pages of 16, heads of 128) down to one (pages of 128, heads of 64), with one, two and more key tiles, a last tile of few rows, and
rows beside the portion that must stay as they are."""
import pytest
import torch
from test_attention_tails import _want

F64 = torch.float64


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("page", [16, 32, 64, 128])
@pytest.mark.parametrize("cached,rows", [(0, 70), (0, 200), (300, 161), (1100, 128)])
def test_pages(cached, rows, page, hd, monkeypatch):
    import kernel_refs as ref
    from tiny_inference_server_b200.kernels import ops
    from tiny_inference_server_b200.kernels.attention_plan import TileSet, plan_tiles
    monkeypatch.setattr(ops, "TC_ATTENTION_MIN_TILES", 1)
    H, KVH, m = 6, 2, cached + rows
    gen = torch.Generator().manual_seed(page + rows)
    bf = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16)  # noqa: E731
    pages = -(-m // page)
    table = torch.randperm(pages + 1, generator=gen)[:pages].to(torch.int32)[None]
    plane = torch.full((pages + 1, 2, KVH, page, hd), float("nan"), dtype=torch.bfloat16)
    plane[table[0].long()] = 0
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
    fault = t([0] * 4)
    out = torch.full((rows + 8, H * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    before = ops.calls["attn_tc"]
    ops.paged_attention(q.cuda(), out[:rows], plane.cuda(), table.cuda(), pos, slot, H, KVH, hd, page, None, fault, Step())
    assert ops.calls["attn_tc"] == before + 1 and int(fault[0]) == 0
    assert bool((out[rows:] == 7.0).all())
    got = out[:rows].view(rows, H, hd).to(F64)
    # bfloat16 probabilities and outputs, 2^-9 each at random over a row of values
    off = (got - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
    assert bool(torch.isfinite(got).all()) and float(off.max()) < 1e-2
