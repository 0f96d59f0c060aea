"""The row kernels around the expert GEMMs at the sizes where their tiles, rounds and vector widths end: routers over many
tokens, the grouping of pairs, the weighted sum.  References in float64 / integers on the CPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64
DTYPES = [torch.float32, torch.bfloat16]


def _setup():
    from pg_b200 import _cabi as cabi
    return cabi, cabi.lib(), cabi.stream()


def _randn(*shape, seed, dtype, std=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * std).to(dtype)


def _check_choice(idx, got_w, choice, weights, top):
    """Chosen indices are the `top` largest of `choice` up to near ties (fp32 dot products: 1e-5), weights 1e-5."""
    want = torch.sort(choice, dim=-1, descending=True, stable=True)[1][:, :top]
    got_c, want_c = torch.gather(choice, 1, idx), torch.gather(choice, 1, want)
    assert float((got_c - want_c).abs().max()) < 1e-5
    assert all(len(set(r.tolist())) == top for r in idx)
    assert float(((got_w - weights(idx)).abs() / weights(idx)).max()) < 1e-5


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,D,E,top,sg", [(512, 264, 16, 2, True), (513, 1024, 5, 5, False), (515, 2048, 18, 2, True),
                                          (700, 136, 33, 4, True), (511, 264, 40, 3, False),
                                          # from 3072 tokens, or 1024 and 32768 experts x width, several tokens per warp
                                          (3072, 264, 16, 2, True), (3073, 1024, 5, 5, False), (3075, 136, 33, 4, True), (1023, 2048, 18, 2, True),
                                          (1026, 2048, 18, 2, True), (1024, 1024, 32, 4, False), (256, 264, 40, 3, True), (257, 264, 40, 3, True)])
def test_softmax_router_tiles(dtype, T, D, E, top, sg):
    cabi, L, st = _setup()
    h, w = _randn(T, D + 8, seed=1, dtype=dtype), _randn(E, D, seed=2, dtype=dtype, std=D ** -0.5)
    corr, wsg = _randn(E, seed=3, dtype=dtype, std=0.01), _randn(D, seed=4, dtype=dtype, std=D ** -0.5)
    dev = [t.cuda() for t in (h, w, corr, wsg)]
    idx, wt = torch.empty(T, top, dtype=torch.int32, device="cuda"), torch.empty(T, top, device="cuda")
    gate = torch.zeros(T, device="cuda")
    cabi.check(L.pg_moe_route(idx.data_ptr(), wt.data_ptr(), gate.data_ptr() if sg else None, dev[0].data_ptr(), D + 8,
                              dev[1].data_ptr(), dev[2].data_ptr(), dev[3].data_ptr() if sg else None, T, D, E, top, 1.5,
                              cabi.DTYPE_CODE[dtype], st))
    x = h[:, :D].to(F64)
    p = torch.softmax(x @ w.to(F64).T, -1)
    i = idx.cpu().long()
    _check_choice(i, wt.cpu().to(F64), p + corr.to(F64), lambda k: 1.5 * torch.gather(p, 1, k), top)
    if sg:
        assert float((gate.cpu().to(F64) - torch.sigmoid(x @ wsg.to(F64))).abs().max()) < 1e-5


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,D,E,top,groups,keep", [(512, 264, 16, 2, 4, 2), (514, 1024, 8, 3, 1, 1), (601, 2048, 24, 4, 3, 2),
                                                    (3074, 264, 16, 2, 4, 2), (1025, 2048, 32, 4, 4, 2), (1024, 2048, 30, 3, 3, 2), (257, 264, 40, 4, 4, 3)])
def test_grouped_router_tiles(dtype, T, D, E, top, groups, keep):
    cabi, L, st = _setup()
    h, w = _randn(T, D, seed=5, dtype=dtype), _randn(E, D, seed=6, dtype=dtype, std=D ** -0.5)
    corr = _randn(E, seed=7, dtype=dtype, std=0.1)
    dev = [t.cuda() for t in (h, w, corr)]
    idx, wt = torch.empty(T, top, dtype=torch.int32, device="cuda"), torch.empty(T, top, device="cuda")
    cabi.check(L.pg_moe_route_grouped(idx.data_ptr(), wt.data_ptr(), dev[0].data_ptr(), D, dev[1].data_ptr(), dev[2].data_ptr(), T, D,
                                      E, top, groups, keep, cabi.DTYPE_CODE[dtype], st))
    s = torch.sigmoid(h.to(F64) @ w.to(F64).T)
    c = s + corr.to(F64)
    gs = c.view(T, groups, -1)
    score = gs.topk(min(2, gs.shape[2]), -1)[0].sum(-1)
    kept = torch.zeros_like(score, dtype=torch.bool).scatter_(1, score.topk(keep, -1)[1], True)
    margin = score.sort(-1, descending=True)[0]
    sure = (margin[:, keep - 1] - margin[:, keep] > 1e-5) if keep < groups else torch.ones(T, dtype=torch.bool)
    c = c.masked_fill(~kept.repeat_interleave(E // groups, 1), -1e3)
    i = idx.cpu().long()

    def weights(k):
        v = torch.gather(s[sure], 1, k)
        return v / v.sum(-1, keepdim=True)
    _check_choice(i[sure], wt.cpu().to(F64)[sure], c[sure], weights, top)


@pytest.mark.parametrize("pairs,top,E,extra", [(1, 1, 1, 0), (255, 1, 3, 1), (256, 2, 16, 0), (258, 2, 600, 2),
                                               (16384, 2, 16, 1), (16386, 2, 16, 1), (40000, 4, 513, 3), (40000, 4, 8, 0)])
def test_grouping_of_pairs(pairs, top, E, extra):
    cabi, L, st = _setup()
    g = torch.Generator().manual_seed(pairs)
    idx = torch.randint(0, E + extra, (pairs,), generator=g, dtype=torch.int32)
    d = idx.cuda()
    off = torch.full((E + 1,), -7, dtype=torch.int32, device="cuda")
    rows = torch.full((pairs,), -7, dtype=torch.int32, device="cuda")
    pos = torch.full((pairs,), -7, dtype=torch.int32, device="cuda")
    cabi.check(L.pg_moe_sort(off.data_ptr(), rows.data_ptr(), pos.data_ptr(), d.data_ptr(), pairs, top, E, st))
    off, rows, pos = off.cpu(), rows.cpu(), pos.cpu()
    routed = idx < E
    want = torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(idx[routed].long(), minlength=E).cumsum(0)])
    assert torch.equal(off.long(), want)
    assert bool((pos[~routed] == -1).all())
    p, e = pos[routed].long(), idx[routed].long()
    assert torch.equal(p.sort()[0], torch.arange(int(routed.sum())))
    assert bool(((p >= want[e]) & (p < want[e + 1])).all())
    assert torch.equal(rows[p].long(), torch.nonzero(routed)[:, 0] // top)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,D,top,shared,pad", [(3, 8, 1, False, 0), (5, 264, 2, True, 8), (67, 2056, 5, True, 0), (9, 250, 4, True, 0)])
def test_weighted_sum(dtype, T, D, top, shared, pad):
    cabi, L, st = _setup()
    g = torch.Generator().manual_seed(11)
    pos = torch.randperm(T * top, generator=g).to(torch.int32)
    pos[torch.randint(0, T * top, (max(1, T // 3),), generator=g)] = -1
    y, h, so = (_randn(n, D + pad, seed=s, dtype=dtype) for n, s in ((T * top, 12), (T, 13), (T, 14)))
    w, sgate, x = torch.rand(T, top, generator=g), torch.rand(T, generator=g), torch.randn(T, D, generator=g)
    dev = [t.cuda() for t in (y, pos, w, h, so, sgate, x)]
    cabi.check(L.pg_moe_combine(dev[6].data_ptr(), dev[0].data_ptr(), D + pad, dev[1].data_ptr(), dev[2].data_ptr(), dev[3].data_ptr(),
                                D + pad, dev[4].data_ptr() if shared else None, D + pad, dev[5].data_ptr() if shared else None, T, D,
                                top, cabi.DTYPE_CODE[dtype], st))
    pl = pos.view(T, top).long()
    src = torch.where((pl >= 0)[..., None], y[pl.clamp_min(0), :D].to(F64), h[:, None, :D].to(F64))
    want = x.to(F64) + (w.to(F64)[..., None] * src).sum(1)
    if shared:
        want += sgate.to(F64)[:, None] * so[:, :D].to(F64)
    # fp32 sums of up to top + 2 terms of size ~3
    assert float((dev[6].cpu().to(F64) - want).abs().max()) < 1e-5
    full = torch.arange(T * top, dtype=torch.int32).cuda()
    out = torch.zeros(T, D + pad, dtype=dtype, device="cuda")
    cabi.check(L.pg_moe_combine_out(out.data_ptr(), D + pad, dev[0].data_ptr(), D + pad, full.data_ptr(), dev[2].data_ptr(),
                                    dev[4].data_ptr() if shared else None, D + pad, T, D, top, cabi.DTYPE_CODE[dtype], st))
    want = (w.to(F64)[..., None] * y[:, :D].to(F64).view(T, top, D)).sum(1) + (so[:, :D].to(F64) if shared else 0.0)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6      # one rounding of the result
    assert bool(((out[:, :D].cpu().to(F64) - want).abs() <= eps * want.abs() + 1e-5).all())
    assert bool((out[:, D:] == 0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["silu", "clamped", "none", "relu2"])
@pytest.mark.parametrize("counts,N,K", [([0, 1, 0, 3], 8, 8), ([2, 0, 9], 24, 72), ([17, 0, 1, 16, 30], 40, 1032), ([1] * 40, 16, 520),
                                        ([0, 0, 12], 1200, 1024), ([5, 11, 0, 0], 2056, 2048)])
def test_few_rows_per_expert(dtype, kind, counts, N, K):
    """Row blocks of up to 16 rows (an expert with more, experts without), features that end inside a unit, columns that end inside
    and behind a chunk of 1024, fewer and more units than CTAs; rows behind the last expert's are not written."""
    cabi, L, st = _setup()
    E, P, dual = len(counts), sum(counts) + 1, kind in ("silu", "clamped")
    off = torch.tensor([0] + counts).cumsum(0).to(torch.int32)
    a, w = _randn(P, K + 8, seed=21, dtype=dtype), _randn(E, (2 if dual else 1) * N, K, seed=22, dtype=dtype, std=K ** -0.5)
    a[-1] = float("nan")                                 # nobody's row
    ad, wd, offd = a.cuda(), w.cuda(), off.cuda()
    out = torch.full((P, N + 8), 7.0, dtype=dtype, device="cuda")
    code = {"silu": cabi.GLU_SILU, "clamped": cabi.GLU_CLAMPED, "none": cabi.GLU_NONE, "relu2": cabi.ACT_RELU2}[kind]
    cabi.check(L.pg_moe_gemm_act(out.data_ptr(), N + 8, ad.data_ptr(), K + 8, None, wd.data_ptr(), offd.data_ptr(), P, E, N, K, code, 1.5, 2,
                                 None, cabi.DTYPE_CODE[dtype], st))
    e = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))
    y = torch.einsum("pk,pnk->pn", a[:-1, :K].to(F64), w.to(F64)[e])
    g, u = y[:, :N], y[:, N:]
    if kind == "silu":
        y = g * torch.sigmoid(g) * u
    elif kind == "clamped":
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
        y = g * torch.sigmoid(1.702 * g) * (u + 1)
    elif kind == "relu2":
        y = g.clamp(min=0) ** 2
    got = out[:-1, :N].cpu().to(F64)
    # up to five roundings of values of about 1, each within half a step of the type
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert float((got - y).norm() / y.norm()) < 2 * eps and float((got - y).abs().max()) < 6 * eps * float(y.abs().max())
    assert bool((out[-1] == 7).all()) and bool((out[:, N:] == 7).all())
