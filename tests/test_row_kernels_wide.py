"""Convolutions whose threads take several rows, and norms of rows in one pass (csrc/seqmix.cu), beside the forms that take fewer rows:
the same inputs in one step of many rows and in steps of few give the same numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from tiny_inference_server_b200.kernels import ops
    return ops


def _rows(lengths, device="cuda"):
    """(row_slot, row_last) of a step of these portions; a length below zero: that many padding rows."""
    slot, last, at = [], [], 0
    for i, n in enumerate(lengths):
        slot += [-1 if n < 0 else i] * abs(n)
        last += [at + abs(n) - 1] * abs(n)
        at += abs(n)
    t = lambda x: torch.tensor(x, dtype=torch.int32, device=device)  # noqa: E731
    return t(slot), t(last)


# one request; portions that begin and end inside a thread's four rows, shorter than the taps, single rows and padding between; a
# number of rows that is no multiple of four; few channels (a row a thread) and so many that a thread takes four
@pytest.mark.parametrize("C", [72, 1808])
@pytest.mark.parametrize("lengths", [[777], [1, 2, 3, 700, 1, 1, 5, 64], [640, -3, 9, 1, -1, 2, 130], [1] * 660])
@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("silu", [False, True])
def test_convolution_of_many_rows(lengths, taps, dtype, silu, C):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(taps)
    n = sum(abs(x) for x in lengths)
    slot, last = _rows(lengths)
    x = torch.randn(n, C + 8, generator=g, device="cuda").to(dtype)[:, :C]
    w = torch.randn(taps, C, generator=g, device="cuda")
    bias = torch.randn(C, generator=g, device="cuda")
    state = torch.randn(len(lengths), (taps - 1) * C, generator=g, device="cuda")
    out, after = torch.full((n, C), 7.0, dtype=dtype, device="cuda"), state.clone()
    ops.causal_conv(x, w, after, out, slot, last, residual=True, silu=silu, bias=bias)
    at = 0
    for i, length in enumerate(lengths):
        rows = slice(at, at + abs(length))
        at += abs(length)
        if length < 0:
            assert bool((out[rows] == 7.0).all())
            continue
        past = torch.cat([state[i].view(taps - 1, C).double(), x[rows].double()])
        y = sum(past[j:j + length] * w[j].double() for j in range(taps)) + bias.double() + x[rows].double()
        y = torch.nn.functional.silu(y) if silu else y
        # taps + 2 roundings of numbers of a few units, and the result's own
        tol = dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=2.0 ** -8, atol=2.0 ** -8)
        torch.testing.assert_close(out[rows].double(), y, **tol)
        assert torch.equal(after[i].view(taps - 1, C), past[len(past) - taps + 1:].float())


# rows of 7 to 1024 vectors; one vector of keys and values a head; without norms, with values of another layer
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,G,kd,vd", [(40, 1, 8, 8), (1536, 3, 128, 128), (264, 2, 24, 40), (2048, 4, 256, 256)])
@pytest.mark.parametrize("norms,mix", [(True, False), (False, True), (True, True)])
def test_norms_in_one_pass(dtype, nq, G, kd, vd, norms, mix):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(nq)
    nk, nv, page, n = G * kd, G * vd, 16, 950
    lengths = [400, -2, 300, 1, 247]
    slot, _ = _rows(lengths)
    pos = torch.cat([torch.arange(abs(x)) for x in lengths]).to(torch.int32).cuda()
    table = torch.randperm(5 * 32, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(5, 32).cuda()
    qkv = torch.randn(n, nq + nk + nv + 8, generator=g, device="cuda").to(dtype)[:, :nq + nk + nv]
    other = torch.randn(n, nv, generator=g, device="cuda").to(dtype) if mix else None
    lam = torch.tensor([0.3], device="cuda") if mix else None
    wq, wk = (torch.randn(m, generator=g, device="cuda") for m in (nq, nk)) if norms else (None, None)
    got = []
    for rows in ([slice(0, n)], [slice(0, 500), slice(500, n)]):            # more rows than the form takes, then fewer
        q = qkv.clone()
        k_pages, v_pages = (torch.zeros(5 * 32, G, page, m, dtype=dtype, device="cuda") for m in (kd, vd))
        fault = torch.zeros(4, dtype=torch.int32, device="cuda")
        for r in rows:
            ops.norm_mix_store(q[r], nq, nk, nv, wq, wk, 1e-6, None if other is None else other[r], lam, k_pages, v_pages, table,
                               pos[r], slot[r], page, fault)
        assert int(fault[0]) == 0
        got.append((q, k_pages, v_pages))
    # the sums of squares are added up in another order, then one rounding of the result
    tol = dict(rtol=1e-5, atol=1e-6) if dtype == torch.float32 else dict(rtol=2.0 ** -7, atol=1e-6)
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, **tol)
    q = got[1][0]
    want = qkv[:, :nq].double()
    if norms:
        want = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-6) * wq.double()
    live = slot >= 0
    torch.testing.assert_close(q[live][:, :nq].double(), want[live], rtol=1e-5 if dtype == torch.float32 else 2.0 ** -7, atol=1e-5)
    assert torch.equal(q[~live], qkv[~live])


# the first row on a 16-byte boundary, and four, eight and twelve bytes behind one; rows of whole vectors and others
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("d", [8, 72, 1536, 12, 7])
def test_embeddings_into_a_view(dtype, shift, d):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(d)
    table = torch.randn(50, d, generator=g, device="cuda").to(dtype)
    tokens = torch.randint(0, 50, (13,), generator=g, device="cuda").to(torch.int32)
    flat = torch.full((13 * d + 8,), 7.0, device="cuda")
    out = flat[shift:shift + 13 * d].view(13, d)
    ops.embed_rows(table, tokens, out, 0.75)
    assert torch.equal(out, table[tokens.long()].float() * 0.75)
    assert bool((flat[:shift] == 7.0).all()) and bool((flat[shift + 13 * d:] == 7.0).all())


# both sides of the limits: by rows (narrow rows), by threads (wide ones); 1024 vectors a row, and more than one pass takes
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,G,kd,vd,counts", [(40, 1, 8, 8, (899, 900)), (3072, 8, 128, 128, (272, 274, 546, 547)), (3072, 8, 64, 64, (341, 342, 683, 684)),
                                               (6144, 8, 128, 128, (341, 342))])
def test_norms_at_the_limits_of_one_pass(dtype, nq, G, kd, vd, counts):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(nq)
    nk, nv, page = G * kd, G * vd, 16
    for n in counts:
        pages = -(-n // page)
        slot, pos = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda")
        table = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()[None]
        qkv = torch.randn(n, nq + nk + nv, generator=g, device="cuda").to(dtype)
        wq, wk = torch.randn(nq, generator=g, device="cuda"), torch.randn(nk, generator=g, device="cuda")
        k_pages, v_pages = (torch.zeros(pages, G, page, m, dtype=dtype, device="cuda") for m in (kd, vd))
        fault, got = torch.zeros(4, dtype=torch.int32, device="cuda"), qkv.clone()
        ops.norm_mix_store(got, nq, nk, nv, wq, wk, 1e-6, None, None, k_pages, v_pages, table, pos, slot, page, fault)
        assert int(fault[0]) == 0
        q, k, v = qkv.double().split([nq, nk, nv], 1)
        # a sum of squares in 32 bits, three products, then the result's own rounding
        tol = dict(rtol=1e-5, atol=1e-6) if dtype == torch.float32 else dict(rtol=2.0 ** -7, atol=1e-6)
        torch.testing.assert_close(got[:, :nq].double(), q / torch.sqrt((q * q).mean(-1, keepdim=True) + 1e-6) * wq.double(), **tol)
        keys = k_pages[table[0].long()].transpose(1, 2).reshape(pages * page, nk)[:n]
        values = v_pages[table[0].long()].transpose(1, 2).reshape(pages * page, nv)[:n]
        torch.testing.assert_close(keys.double(), k / torch.sqrt((k * k).mean(-1, keepdim=True) + 1e-6) * wk.double(), **tol)
        assert torch.equal(values, v.to(dtype))
