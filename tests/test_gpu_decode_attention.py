"""Decode attention of 256-wide heads in 16-bit types at the edges of its 16-token chunks, pages, warps and cluster sizes,
against float64 with the scores rounded to the model type as the reference materialises them."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("dtype,rel", [(torch.bfloat16, 4e-3), (torch.float16, 6e-4)])
@pytest.mark.parametrize("B,T,G,nkv,page", [(1, 1, 8, 1, 64), (1, 16, 8, 1, 16), (2, 17, 8, 1, 64), (3, 65, 4, 2, 64), (1, 262, 8, 1, 64),
                                            (1, 1025, 2, 1, 32), (19, 130, 8, 1, 64), (40, 31, 1, 3, 64), (80, 257, 8, 1, 64),
                                            (150, 48, 8, 1, 64), (2, 2100, 8, 1, 64)])
def test_chunks_pages_and_clusters(dtype, rel, B, T, G, nkv, page):
    from pg_b200 import _cabi as cabi
    hd, nq = 256, G * nkv
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + T)
    new = lambda *s: torch.randn(s, device="cuda", generator=g).to(dtype)  # noqa: E731
    lens = torch.randint(max(1, T - 40), T + 1, (B,), device="cuda", generator=g)
    lens[0] = T
    cols = -(-T // page)
    pages = B * cols + 2
    kp, vp, q = new(pages, page, nkv * hd), new(pages, page, nkv * hd), new(B, nq * hd)
    pt = torch.randperm(pages, device="cuda", generator=g)[:B * cols].to(torch.int32).view(B, cols)
    out = torch.zeros(B, nq * hd, dtype=dtype, device="cuda")
    kvl = (lens - 1).to(torch.int32)
    cabi.check(cabi.lib().pg_decode_attention(out.data_ptr(), q.data_ptr(), kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), cols, page,
                                              kvl.data_ptr(), 1, B, nq, nkv, hd, math.sqrt(hd), None, None, 0, cabi.DTYPE_CODE[dtype],
                                              cabi.stream()))
    for b in sorted({0, B // 2, B - 1}):
        n = int(lens[b])
        k, v = (p[pt[b].long()].reshape(-1, nkv, hd)[:n].to(F64).repeat_interleave(G, 1) for p in (kp, vp))
        s = torch.einsum("hd,nhd->hn", q[b].view(nq, hd).to(F64), k).to(dtype).to(F64) / math.sqrt(hd)
        want = torch.einsum("hn,nhd->hd", torch.softmax(s, -1), v).reshape(-1)
        got = out[b].to(F64)
        # one rounding of the result (2^-9 and 2^-12 relative at most) and the odd score that rounds the other way
        assert float((got - want).norm() / want.norm()) < rel


@pytest.mark.parametrize("T,lo,hi", [(262, 0, 16), (262, 32, 70), (1345, 1024, 1345), (600, 5, 600), (40, 0, 40)])
def test_scores_below_the_type(T, lo, hi):
    """fp16 scores of the tokens [lo, hi) round to -inf for half of the heads: those tokens weigh nothing there, wherever
    the chunks, warps and clusters cut, and a head without any other token is undefined."""
    from pg_b200 import _cabi as cabi
    hd, G, page, dt = 256, 8, 64, torch.float16
    g = torch.Generator(device="cuda").manual_seed(T + lo)
    cols = -(-T // page)
    kp, vp = ((torch.randn(cols, page, hd, device="cuda", generator=g) * std).to(dt) for std in (0.01, 1.0))
    q = (torch.randn(G, hd, device="cuda", generator=g) * 0.3).to(dt)
    kp.view(-1, hd)[lo:hi] = -30.0
    q[::2] = 30.0
    pt = torch.arange(cols, dtype=torch.int32, device="cuda")
    out, kvl = torch.zeros(G, hd, dtype=dt, device="cuda"), torch.tensor([T], dtype=torch.int32, device="cuda")
    cabi.check(cabi.lib().pg_decode_attention(out.data_ptr(), q.data_ptr(), kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), cols, page,
                                              kvl.data_ptr(), 0, 1, G, 1, hd, 16.0, None, None, 0, cabi.PG_F16, cabi.stream()))
    k, v = (p.view(-1, hd)[:T].to(F64) for p in (kp, vp))
    want = torch.softmax((q.to(F64) @ k.T).to(dt).to(F64) / 16.0, -1) @ v
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and bool(torch.isnan(want).any()) == (hi - lo == T)
    sure = ~torch.isnan(want)
    assert float((out.to(F64) - want)[sure].norm() / want[sure].norm()) < 6e-4      # as above


@pytest.mark.parametrize("dtype,rel", [(torch.bfloat16, 4e-3), (torch.float16, 6e-4)])
@pytest.mark.parametrize("T,low", [(4097, -15.0), (700, -11.5), (65, -9.25)])
def test_many_small_weights(dtype, rel, T, low):
    """One token of weight 1 and value 0, T - 1 of weight exp(low) and value 1: the small weights make up the result."""
    from pg_b200 import _cabi as cabi
    hd, G, page = 256, 8, 64
    cols = -(-T // page)
    kp, vp = torch.zeros(cols, page, hd, dtype=dtype, device="cuda"), torch.ones(cols, page, hd, dtype=dtype, device="cuda")
    kp.view(-1, hd)[1:, 0] = 16.0 * low
    vp.view(-1, hd)[0] = 0.0
    q = torch.zeros(G, hd, dtype=dtype, device="cuda")
    q[:, 0] = 1.0
    pt = torch.arange(cols, dtype=torch.int32, device="cuda")
    out, kvl = torch.zeros(G, hd, dtype=dtype, device="cuda"), torch.tensor([T], dtype=torch.int32, device="cuda")
    cabi.check(cabi.lib().pg_decode_attention(out.data_ptr(), q.data_ptr(), kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), cols, page,
                                              kvl.data_ptr(), 0, 1, G, 1, hd, 16.0, None, None, 0, cabi.DTYPE_CODE[dtype], cabi.stream()))
    small = (T - 1) * math.exp(low)
    assert float((out.to(F64) / (small / (1.0 + small)) - 1.0).abs().max()) < rel     # one rounding of the result


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T", [1, 37, 262, 1345])
def test_infinite_values(dtype, T):
    """An infinity in a value row makes its column infinite for every head that gives the token weight, and no other column."""
    from pg_b200 import _cabi as cabi
    hd, G, page = 256, 8, 64
    g = torch.Generator(device="cuda").manual_seed(T)
    cols = -(-T // page)
    kp, vp, q = (torch.randn(s, device="cuda", generator=g).to(dtype) * std for s, std in (((cols, page, hd), 0.3), ((cols, page, hd), 1.0),
                                                                                          ((G, hd), 0.3)))
    for token, col, value in ((0, 3, math.inf), (T // 2, 130, -math.inf), (T - 1, 70, math.inf)):
        vp.view(-1, hd)[token, col] = value
    pt = torch.arange(cols, dtype=torch.int32, device="cuda")
    out, kvl = torch.zeros(G, hd, dtype=dtype, device="cuda"), torch.tensor([T], dtype=torch.int32, device="cuda")
    cabi.check(cabi.lib().pg_decode_attention(out.data_ptr(), q.data_ptr(), kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), cols, page,
                                              kvl.data_ptr(), 0, 1, G, 1, hd, 16.0, None, None, 0, cabi.DTYPE_CODE[dtype], cabi.stream()))
    k, v = (p.view(-1, hd)[:T].to(F64) for p in (kp, vp))
    w = torch.softmax((q.to(F64) @ k.T).to(dtype).to(F64) / 16.0, -1)
    fine = torch.isfinite(v).all(0)
    assert bool((out[:, 3] == math.inf).all()) and bool((out[:, 130] == -math.inf).all()) and bool((out[:, 70] == math.inf).all())
    want = w @ v[:, fine]
    assert float((out[:, fine].to(F64) - want).norm() / want.norm()) < 4e-3      # the bound of bf16 above


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,T,G,nkv,page,hd", [(1, 1, 8, 1, 64, 256), (1, 17, 1, 2, 16, 256), (3, 64, 4, 2, 64, 256), (15, 257, 8, 1, 32, 256),
                                               (40, 49, 2, 1, 64, 256), (80, 130, 8, 1, 64, 256), (150, 33, 8, 1, 64, 256),
                                               (2, 40, 4, 1, 20, 256), (2, 33, 4, 1, 16, 64)])
def test_rotary_and_append_inside(dtype, B, T, G, nkv, page, hd):
    """One call leaves the outputs and the cache that rotary embedding + append and the attention leave as two, bit for bit."""
    from pg_b200 import _cabi as cabi
    L, nq, max_pos = cabi.lib(), G * nkv, 512
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + T)
    new = lambda *s: torch.randn(s, device="cuda", generator=g).to(dtype)  # noqa: E731
    kvl = torch.randint(max(0, T - 40), T, (B,), device="cuda", generator=g).to(torch.int32)
    kvl[0] = T - 1
    pos = torch.randint(-1, max_pos + 2, (B,), device="cuda", generator=g).to(torch.int32)   # the ends are clamped
    cols = -(-T // page)
    pages = B * cols + 2
    pt = torch.randperm(pages, device="cuda", generator=g)[:B * cols].to(torch.int32).view(B, cols)
    pools, qkv = [new(pages, page, nkv * hd) for _ in "kv"], new(B, (nq + 2 * nkv) * hd)
    freq = 1.0 / 10000 ** (torch.arange(0, hd, 2, device="cuda").float() / hd)
    code, st, scale = cabi.DTYPE_CODE[dtype], cabi.stream(), math.sqrt(hd)
    results = []
    for one_call in (False, True):
        kp, vp = (p.clone() for p in pools)
        q, out = torch.zeros(B, nq * hd, dtype=dtype, device="cuda"), torch.zeros(B, nq * hd, dtype=dtype, device="cuda")
        where = (kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), cols, page, kvl.data_ptr())
        if one_call:
            cabi.check(L.pg_decode_attention_rope(out.data_ptr(), q.data_ptr(), qkv.data_ptr(), freq.data_ptr(), pos.data_ptr(), *where,
                                                  B, nq, nkv, hd, max_pos, scale, code, st))
        else:
            cabi.check(L.pg_rope_append(q.data_ptr(), qkv.data_ptr(), freq.data_ptr(), pos.data_ptr(), *where, B, 1, nq, nkv, hd,
                                        max_pos, code, st))
            cabi.check(L.pg_decode_attention(out.data_ptr(), q.data_ptr(), *where, 1, B, nq, nkv, hd, scale, None, None, 0, code, st))
        results.append((out, kp, vp))
    assert all(torch.equal(a, b) for a, b in zip(*results))


def _rotated(rows, freq, pos, dtype):
    """The rotary embedding's products and sums, each rounded to the type.  rows [B, heads, hd]."""
    ang = pos.clamp(min=0)[:, None, None].float() * freq
    c, s = ang.cos().to(dtype), ang.sin().to(dtype)
    x, y = rows.chunk(2, -1)
    return torch.cat([x * c + -y * s, y * c + x * s], -1)


@pytest.mark.parametrize("dtype,rel", [(torch.bfloat16, 4e-3), (torch.float16, 6e-4)])
@pytest.mark.parametrize("B,T,G,page", [(1, 1, 8, 64), (2, 37, 8, 64), (3, 262, 4, 16), (1, 1345, 2, 64), (80, 100, 8, 64)])
def test_infinite_values_behind_a_rotation(dtype, rel, B, T, G, page):
    """The same with the rotation and the new row inside, the last infinity in the new row, against float64."""
    from pg_b200 import _cabi as cabi
    hd = 256
    g = torch.Generator(device="cuda").manual_seed(B + T)
    new = lambda *s: torch.randn(s, device="cuda", generator=g).to(dtype)  # noqa: E731
    cols = -(-T // page)
    pages = B * cols
    kp, vp, qkv = new(pages, page, hd) * 0.3, new(pages, page, hd), new(B, G + 2, hd) * 0.3
    pt = torch.randperm(pages, device="cuda", generator=g).to(torch.int32).view(B, cols)
    kvl, pos = (torch.full((B,), n, dtype=torch.int32, device="cuda") for n in (T - 1, 41))
    freq = 1.0 / 10000 ** (torch.arange(0, hd, 2, device="cuda").float() / hd)
    for token, col, value in ((0, 3, math.inf), (T // 2, 130, -math.inf)):
        if token < T - 1:
            vp[pt[:, token // page].long(), token % page, col] = value
        else:
            qkv[:, G + 1, col] = value
    qkv[:, G + 1, 70] = math.inf
    q, out = torch.zeros(B, G * hd, dtype=dtype, device="cuda"), torch.zeros(B, G, hd, dtype=dtype, device="cuda")
    cabi.check(cabi.lib().pg_decode_attention_ex(out.data_ptr(), q.data_ptr(), kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), cols, page, pages,
                                                 kvl.data_ptr(), 1, B, G, 1, hd, 16.0, qkv.data_ptr(), freq.data_ptr(), pos.data_ptr(), 512,
                                                 cabi.DTYPE_CODE[dtype], cabi.stream()))
    turned = _rotated(qkv[:, :G + 1], freq, pos, dtype)
    for b in sorted({0, B // 2, B - 1}):
        k, v = (torch.cat([p[pt[b].long()].reshape(-1, hd)[:T - 1], row]).to(F64) for p, row in ((kp, turned[b, G:]), (vp, qkv[b, G + 1:])))
        w = torch.softmax((turned[b, :G].to(F64) @ k.T).to(dtype).to(F64) / 16.0, -1)
        fine, o = torch.isfinite(v).all(0), out[b]
        assert bool((o[:, 3] == math.inf).all()) and bool((o[:, 130] == -math.inf).all()) and bool((o[:, 70] == math.inf).all())
        want = w @ v[:, fine]
        assert float((o[:, fine].to(F64) - want).norm() / want.norm()) < rel           # the bound of finite values above


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,counted", [(1, 61, "all"), (8, 257, "all"), (8, 257, "one"), (8, 257, "none"), (40, 15, "all")])
def test_steps_follow_one_another(dtype, B, T, counted):
    """A captured step whose lengths and positions are moved on in front of it, replayed: what is read ahead of the launch before is
    read again behind it, whether the table's pages are known to be the pool's or not.  Against the two launches, bit for bit."""
    from pg_b200 import _cabi as cabi
    L, hd, G, page, steps = cabi.lib(), 256, 8, 16, 5
    g = torch.Generator(device="cuda").manual_seed(B + T)
    new = lambda *s: torch.randn(s, device="cuda", generator=g).to(dtype)  # noqa: E731
    cols = -(-(T + steps) // page)
    pages = B * cols
    pt = torch.randperm(pages, device="cuda", generator=g).to(torch.int32).view(B, cols)
    pools, qkv, w = [new(pages, page, hd) for _ in "kv"], new(B, (G + 2) * hd), new(1152)
    freq = 1.0 / 10000 ** (torch.arange(0, hd, 2, device="cuda").float() / hd)
    kvl, pos = (torch.full((B,), n, dtype=torch.int32, device="cuda") for n in (T - 2, T + 6))
    ids, keys = torch.zeros(B, dtype=torch.int64, device="cuda"), torch.zeros(B, dtype=torch.int64, device="cuda")
    x, y = new(B, 1152), new(B, 1152)
    q, out = torch.zeros(B, G * hd, dtype=dtype, device="cuda"), torch.zeros(B, G * hd, dtype=dtype, device="cuda")
    (kp, vp), (kr, vr) = pools, [torch.empty_like(p) for p in pools]
    qr, want = torch.zeros_like(q), torch.zeros_like(out)
    code, num = cabi.DTYPE_CODE[dtype], {"all": pages, "one": 1, "none": 0}[counted]

    def step():
        st = cabi.stream()
        cabi.check(L.pg_step_advance(ids.data_ptr(), None, 0, None, keys.data_ptr(), ids.data_ptr(), kvl.data_ptr(), pos.data_ptr(), B, None, st))
        cabi.check(L.pg_rmsnorm(y.data_ptr(), x.data_ptr(), w.data_ptr(), B, 1152, 1e-6, code, st))   # lets the next launch start early
        cabi.check(L.pg_decode_attention_ex(out.data_ptr(), q.data_ptr(), kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), cols, page, num,
                                            kvl.data_ptr(), 1, B, G, 1, hd, 16.0, qkv.data_ptr(), freq.data_ptr(), pos.data_ptr(), 512, code, st))
    step()
    for ref, pool in ((kr, kp), (vr, vp)):
        ref.copy_(pool)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        step()
    for _ in range(steps):
        graph.replay()
        st, where = cabi.stream(), (kr.data_ptr(), vr.data_ptr(), pt.data_ptr(), cols, page, kvl.data_ptr())
        cabi.check(L.pg_rope_append(qr.data_ptr(), qkv.data_ptr(), freq.data_ptr(), pos.data_ptr(), *where, B, 1, G, 1, hd, 512, code, st))
        cabi.check(L.pg_decode_attention(want.data_ptr(), qr.data_ptr(), *where, 1, B, G, 1, hd, 16.0, None, None, 0, code, st))
        assert torch.equal(out, want) and torch.equal(kp, kr) and torch.equal(vp, vr)
        qkv.copy_(new(B, (G + 2) * hd))
    assert int(kvl[0]) == T - 1 + steps
