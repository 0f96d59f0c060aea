"""The tensor-core kernels at the edges of their tiles, clusters and splits, against float64 products of the same 16-bit
operands with the rounding points of the epilogues."""
import ctypes
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
F64 = torch.float64
BF = torch.bfloat16
TYPES = [BF, torch.float16]


def _cabi():
    from pg_b200 import _cabi as cabi
    return cabi, cabi.lib(), cabi.stream()


def _randn(gen, *shape, std=1.0, dtype=BF):
    return (torch.randn(shape, device="cuda", generator=gen) * std).to(dtype)


def _rel(got, want):
    return float((got.to(F64) - want).norm() / want.norm())


def _tol(dtype, bf16, tanh=False):
    """The same roundings cost fp16 an eighth of bf16's; the hardware tanh (2^-11) stays what it is."""
    return bf16 if dtype == BF else bf16 / 8 + (2.0 ** -11 if tanh else 0.0)


def _gelu(x):
    return F.gelu(x, approximate="tanh")


# bf16 results: every rounding adds at most 2^-9 relative (rms about 2^-10.8), the hardware tanh 2^-11: three roundings of
# a pairing stay below 4e-3
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("epi", ["geglu", "swiglu"])
@pytest.mark.parametrize("M,N,K", [(1292, 2048, 256), (1100, 2056, 128), (513, 4096, 72), (385, 8200, 64)])
def test_gated_pairs(epi, M, N, K, dtype):
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(M)
    a, w = _randn(g, M, K, dtype=dtype), _randn(g, 2 * N, K, std=K ** -0.5, dtype=dtype)
    out = torch.zeros(M + 1, N, dtype=dtype, device="cuda")
    cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), None, None, M, N, K, K, K, N, 0, 0,
                         cabi.EPI_GEGLU if epi == "geglu" else cabi.EPI_SWIGLU, 0, 2, cabi.DTYPE_CODE[dtype], st))
    z = a.to(F64) @ w.to(F64).T
    want = (_gelu(z[:, :N]) if epi == "geglu" else F.silu(z[:, :N])) * z[:, N:]
    assert _rel(out[:M], want) < _tol(dtype, 5e-3, epi == "geglu")
    assert bool((out[M] == 0).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("M,N,K", [(1292, 2048, 512), (1292, 2560, 200), (700, 2048, 1024), (1025, 264, 4096)])
def test_row_major_pairs_with_residual(M, N, K, dtype):
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(N)
    a, w, r = _randn(g, M, K, dtype=dtype), _randn(g, N, K, std=K ** -0.5, dtype=dtype), _randn(g, M, N, dtype=dtype)
    out = torch.zeros(M + 1, N, dtype=dtype, device="cuda")
    cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), None, r.data_ptr(), M, N, K, K, K, N, N, 0, cabi.EPI_RES, 0, 2,
                         cabi.DTYPE_CODE[dtype], st))
    assert _rel(out[:M], a.to(F64) @ w.to(F64).T + r.to(F64)) < _tol(dtype, 4e-3)
    assert bool((out[M] == 0).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("M", [4, 8, 31, 32, 33, 64])
@pytest.mark.parametrize("N,K,epi", [(2048, 16384, "res"), (2048, 2048, "res"), (2560, 2048, "none"), (2056, 2048, "bias"), (2048, 4104, "res")])
def test_few_rows_split_over_clusters(M, N, K, epi, dtype):
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a, w = _randn(g, M, K, dtype=dtype), _randn(g, N, K, std=K ** -0.5, dtype=dtype)
    r, b = _randn(g, M, N, dtype=dtype), _randn(g, N, dtype=dtype)
    out = torch.zeros(M + 1, N, dtype=dtype, device="cuda")
    code = {"res": cabi.EPI_RES, "none": cabi.EPI_NONE, "bias": cabi.EPI_BIAS}[epi]
    cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), b.data_ptr() if epi == "bias" else None,
                         r.data_ptr() if epi == "res" else None, M, N, K, K, K, N, N if epi == "res" else 0, 0, code, 0, 0, cabi.DTYPE_CODE[dtype], st))
    want = a.to(F64) @ w.to(F64).T + (r.to(F64) if epi == "res" else b.to(F64) if epi == "bias" else 0.0)
    assert _rel(out[:M], want) < _tol(dtype, 4e-3)
    assert bool((out[M] == 0).all())


def _route(L, M, N, K, epi, f32):
    """The kernel that pg_gemm (impl 0) takes, by the library's own rules (C++ functions of namespace pg)."""
    def rule(name, *args, kind=ctypes.c_bool):
        f = getattr(L, f"_ZN2pg{len(name)}{name}E" + "i" * len(args))
        f.argtypes, f.restype = [ctypes.c_int] * len(args), kind
        return f(*args)
    if rule("gemm_tc_swap_wanted", M, N, K, epi, f32, 0):
        return "pairs"
    if rule("gemm_stream_wanted", M, N, K, epi):
        return "stream"
    if rule("gemm_tc_skinny_wanted", M, N, K, epi):
        return "skinny %d" % rule("gemm_tc_skinny_split", N, K, epi, kind=ctypes.c_int)
    return "split %d" % rule("gemm_tc_splitk_factor", M, N, K, epi, kind=ctypes.c_int)


# partial sums of a split over K change hands by whole row pieces: row tiles with missing rows, feature tiles with missing columns,
# every number of CTAs that share a tile, rows past 256 in a second token tile; results have the roundings of the products above, fp32
# ones too (the type's values, widened)
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("route,M,N,K,epi,f32", [
    ("split 4", 33, 1152, 4304, "res", 0), ("split 2", 129, 1152, 1152, "none", 0), ("split 4", 257, 1160, 4304, "bias_res", 0),
    ("split 4", 256, 1152, 4304, "res", 0), ("split 2", 260, 2048, 2048, "res", 0), ("split 4", 353, 520, 4096, "none", 1),
    ("split 2", 161, 2056, 2048, "none", 1), ("split 2", 384, 1152, 1152, "bias_gelu", 0), ("split 2", 65, 4304, 1152, "bias", 0),
    ("skinny 8", 32, 2056, 16384, "res", 0), ("skinny 8", 17, 2048, 4096, "none", 1), ("skinny 8", 64, 2056, 8192, "res", 0),
    ("skinny 4", 19, 3080, 2048, "none", 0), ("skinny 4", 31, 3080, 2048, "bias_res", 0), ("skinny 4", 50, 3080, 8192, "res", 0),
    ("skinny 4", 25, 3080, 2048, "bias", 1), ("skinny 4", 20, 2432, 1280, "res", 0), ("skinny 2", 5, 9608, 512, "res", 0),
    ("skinny 2", 18, 4304, 1152, "bias_gelu", 0), ("skinny 2", 30, 8200, 2048, "none", 1), ("skinny 2", 60, 8200, 4096, "none", 0),
    ("pairs", 256, 264, 4096, "res", 0), ("pairs", 257, 2048, 16384, "res", 0), ("pairs", 271, 1000, 2048, "none", 0),
    ("pairs", 273, 264, 4096, "res", 0), ("pairs", 384, 2056, 2048, "geglu", 0), ("pairs", 449, 2048, 8192, "res", 0),
    ("pairs", 511, 136, 8192, "res", 0)])
def test_partial_sums_change_hands(gemm_workspace, route, M, N, K, epi, f32, dtype):
    cabi, L, st = _cabi()
    code, pairs = getattr(cabi, "EPI_" + epi.upper()), route == "pairs"
    if not pairs:
        cabi.check(L.pg_set_workspace(None, 0))
        assert _route(L, M, N, K, code, f32) == route
    g = torch.Generator(device="cuda").manual_seed(M + N)
    rows = 2 * N if epi == "geglu" else N
    a, w = _randn(g, M, K, dtype=dtype), _randn(g, rows, K, std=K ** -0.5, dtype=dtype)
    r, b = _randn(g, M, N, dtype=dtype), _randn(g, N, dtype=dtype)
    out = torch.zeros((M + 1) * N, dtype=torch.float32 if f32 else dtype, device="cuda").view(M + 1, N)
    before = cabi.launch_count()
    cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), b.data_ptr() if "bias" in epi else None,
                         r.data_ptr() if "res" in epi else None, M, N, K, K, K, N, N if "res" in epi else 0, 0, code, f32,
                         3 if pairs else 0, cabi.DTYPE_CODE[dtype], st))
    assert cabi.launch_count() - before == (2 if pairs else 1)                 # the pairs' reduction is a launch of its own
    z = a.to(F64) @ w.to(F64).T + (b.to(F64) if "bias" in epi else 0.0)
    want = _gelu(z[:, :N]) * z[:, N:] if epi == "geglu" else _gelu(z) if "gelu" in epi else z + r.to(F64) if "res" in epi else z
    assert _rel(out[:M], want) < _tol(dtype, 5e-3 if epi == "geglu" else 4e-3, "g" in epi)
    assert bool((out[M] == 0).all())


# More weight tiles than CTA pairs (74), the last of them of at most 128 features: a pair's second item, in which one CTA has nothing to
# store, with so short a K that the first item's last store may still be under way.  Every repetition has to give the same bits.
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("impl,M,N,K,epi", [(0, 100, 19008, 64, "res"), (0, 65, 19072, 256, "res"), (3, 128, 9536, 64, "geglu"),
                                            (3, 300, 18952, 64, "none"), (3, 33, 37960, 128, "res")])
def test_a_half_empty_tile_behind_a_whole_one(gemm_workspace, impl, M, N, K, epi, dtype):
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(M)
    rows = 2 * N if epi == "geglu" else N
    assert -(-rows // 256) > 74 and 1 <= rows % 256 <= 128
    a, w = _randn(g, M, K, dtype=dtype), _randn(g, rows, K, std=K ** -0.5, dtype=dtype)
    r = _randn(g, M, N, dtype=dtype)
    code = {"res": cabi.EPI_RES, "none": cabi.EPI_NONE, "geglu": cabi.EPI_GEGLU}[epi]
    z = a.to(F64) @ w.to(F64).T
    want = _gelu(z[:, :N]) * z[:, N:] if epi == "geglu" else z + r.to(F64) if epi == "res" else z
    first = None
    for _ in range(24):
        gemm_workspace.fill_(0xff)                                             # NaN where nothing is stored
        out = torch.zeros(M + 1, N, dtype=dtype, device="cuda")
        before = cabi.launch_count()
        cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), None, r.data_ptr() if epi == "res" else None, M, N, K, K, K, N,
                             N if epi == "res" else 0, 0, code, 0, impl, cabi.DTYPE_CODE[dtype], st))
        assert cabi.launch_count() - before == 2                               # the pair kernel and its reduction
        if first is None:
            first = out
            assert _rel(out[:M], want) < _tol(dtype, 5e-3 if epi == "geglu" else 4e-3, epi == "geglu")
            assert bool((out[M] == 0).all())
        assert torch.equal(out, first)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("act,rel", [("none", 4e-3), ("silu", 5e-3), ("clamped", 6e-3), ("relu2", 6e-3)])
@pytest.mark.parametrize("rows", [[1200, 0, 257, 1], [256, 256, 512, 1024], [3000, 5], [3, 1, 0, 2, 0, 1, 4, 5]])
def test_grouped_products(act, rel, rows, dtype):
    """Experts with many rows (CTA pairs), with none, with one, with a row behind a full tile; a handful of rows in all."""
    cabi, L, st = _cabi()
    E, N, K, P = len(rows), 328, 192, sum(rows)
    g = torch.Generator(device="cuda").manual_seed(P)
    dual = act in ("silu", "clamped")
    a, w = _randn(g, P, K, dtype=dtype), _randn(g, E, 2 * N if dual else N, K, std=K ** -0.5, dtype=dtype)
    off = torch.tensor([sum(rows[:e]) for e in range(E + 1)], dtype=torch.int32, device="cuda")
    out = torch.zeros(P + 1, N, dtype=dtype, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    code = {"none": cabi.GLU_NONE, "silu": cabi.GLU_SILU, "clamped": cabi.GLU_CLAMPED, "relu2": cabi.ACT_RELU2}[act]
    cabi.check(L.pg_moe_gemm_act(out.data_ptr(), N, a.data_ptr(), K, None, w.data_ptr(), off.data_ptr(), P, E, N, K, code, 1.5, 2,
                                 err.data_ptr(), cabi.DTYPE_CODE[dtype], st))
    want = torch.empty(P, N, dtype=F64, device="cuda")
    for e in range(E):
        z = a[off[e]:off[e + 1]].to(F64) @ w[e].to(F64).T
        if act == "silu":
            z = F.silu(z[:, :N]) * z[:, N:]
        elif act == "clamped":
            gt, up = z[:, :N].clamp(max=1.5), z[:, N:].clamp(-1.5, 1.5)
            z = gt * torch.sigmoid(1.702 * gt) * (up + 1.0)
        elif act == "relu2":
            z = z.clamp_min(0.0) ** 2
        want[off[e]:off[e + 1]] = z
    assert int(err) == 0
    assert _rel(out[:P], want) < _tol(dtype, rel)
    assert bool((out[P] == 0).all())


@pytest.mark.parametrize("B,q,T,H,G,hd", [(1, 16, 16, 8, 1, 256), (2, 130, 193, 8, 1, 256), (1, 260, 260, 8, 1, 256), (1, 33, 1000, 4, 2, 256),
                                          (3, 128, 64, 2, 2, 256)])
def test_prompt_attention(B, q, T, H, G, hd):
    """Unmasked attention over pages; scores that grow along the sequence, so that the reference maximum has to follow."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(T)
    cols = -(-T // 64)
    pages = B * cols + 1
    kp, vp, qq = _randn(g, pages, 64, G * hd), _randn(g, pages, 64, G * hd), _randn(g, B * q, H * hd)
    pt = torch.randperm(pages, device="cuda", generator=g)[:B * cols].to(torch.int32).view(B, cols)
    for b in range(B):
        for c in range(cols):
            kp[pt[b, c].long()] *= 0.2 + 1.2 * c
    kvl = torch.full((B,), T - q if T >= q else 0, dtype=torch.int32, device="cuda")
    add = T - int(kvl[0])
    out = torch.zeros(B * q, H * hd, dtype=BF, device="cuda")
    cabi.check(L.pg_attention_tc(out.data_ptr(), H * hd, qq.data_ptr(), B * q, H * hd, 0, kp.data_ptr(), vp.data_ptr(), pages * 64,
                                 G * hd, 0, 0, hd, 0, pt.data_ptr(), cols, 64, kvl.data_ptr(), 0, add, B, q, H, G, hd, math.sqrt(hd),
                                 1, cabi.PG_BF16, st))
    for b in range(B):
        k, v = (p[pt[b].long()].reshape(-1, G, hd)[:T].to(F64).repeat_interleave(H // G, 1) for p in (kp, vp))
        s = torch.einsum("qhd,nhd->hqn", qq[b * q:(b + 1) * q].view(q, H, hd).to(F64), k).to(BF).to(F64) / math.sqrt(hd)
        want = torch.einsum("hqn,nhd->qhd", torch.softmax(s, -1), v).reshape(q, H * hd)
        # weights and result are rounded to bf16 (2^-9 each at most); a score that rounds the other way moves its weight
        assert _rel(out[b * q:(b + 1) * q], want) < 8e-3


@pytest.mark.parametrize("q,T,low", [(3, 70, 64), (130, 260, 128), (16, 200, 130), (5, 40, 40)])
def test_prompt_attention_scores_below_the_type(q, T, low):
    """The first `low` scores of some rows round to -inf in fp16: those keys weigh nothing, and only a row without any other
    key is undefined, as the reference's softmax has it."""
    cabi, L, st = _cabi()
    H, hd, dt = 4, 256, torch.float16
    g = torch.Generator(device="cuda").manual_seed(T + low)
    cols = -(-T // 64)
    kp, vp, qq = (_randn(g, *s, std=std, dtype=dt) for s, std in (((cols, 64, hd), 0.01), ((cols, 64, hd), 1.0), ((q, H * hd), 0.3)))
    kp.view(-1, hd)[:low] = -30.0
    qq.view(q, H, hd)[::2, 1:] = 30.0            # 256 x 30 x -30: below -65504
    pt = torch.arange(cols, dtype=torch.int32, device="cuda").view(1, cols)
    kvl = torch.full((1,), T - q, dtype=torch.int32, device="cuda")
    out = torch.zeros(q, H * hd, dtype=dt, device="cuda")
    cabi.check(L.pg_attention_tc(out.data_ptr(), H * hd, qq.data_ptr(), q, H * hd, 0, kp.data_ptr(), vp.data_ptr(), cols * 64, hd, 0, 0, hd,
                                 0, pt.data_ptr(), cols, 64, kvl.data_ptr(), 0, q, 1, q, H, 1, hd, math.sqrt(hd), 1, cabi.PG_F16, st))
    k, v = (p.view(-1, hd)[:T].to(F64) for p in (kp, vp))
    s = torch.einsum("qhd,nd->hqn", qq.view(q, H, hd).to(F64), k).to(dt).to(F64) / math.sqrt(hd)
    assert bool(torch.isinf(s).any())
    want = torch.einsum("hqn,nd->qhd", torch.softmax(s, -1), v).reshape(q, H * hd)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and bool(torch.isnan(want).any()) == (low == T)
    sure = ~torch.isnan(want)
    # weights and result are rounded to fp16 (2^-12 each at most); a score that rounds the other way moves its weight
    assert float((out.to(F64) - want)[sure].norm() / want[sure].norm()) < 2e-3


@pytest.mark.parametrize("dim,vdim,H,G", [(64, 64, 4, 4), (128, 128, 16, 4), (128, 128, 12, 1), (256, 256, 8, 1), (256, 192, 5, 1)])
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("window,keep,chunk", [(0, 0, 0), (33, 0, 0), (100, 7, 0), (0, 0, 48)])
def test_single_tokens_over_the_cache(dim, vdim, H, G, window, keep, chunk, dtype):
    """Decode-sized ragged steps: positions at the edges of 16-key chunks, pages, windows, blocks and clusters."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(dim + H)
    pos = [0, 1, 15, 16, 17, 63, 64, 127, 500, 1535]
    n, cols = len(pos), 24
    pages = n * cols + 1
    kp, vp = _randn(g, pages, 64, G * dim, dtype=dtype), _randn(g, pages, 64, G * vdim, dtype=dtype)
    q, gate = _randn(g, n, H * dim, dtype=dtype), _randn(g, n, H * vdim, dtype=dtype)
    pt = torch.randperm(pages, device="cuda", generator=g)[:n * cols].to(torch.int32).view(n, cols)
    slopes, sink = torch.rand(H, device="cuda", generator=g) * 0.1, torch.randn(H, device="cuda", generator=g)
    slot, tp = torch.arange(n, dtype=torch.int32, device="cuda"), torch.tensor(pos, dtype=torch.int32, device="cuda")
    out = torch.zeros(n, H * vdim, dtype=dtype, device="cuda")
    cabi.check(L.pg_attention_ragged_masked(out.data_ptr(), H * vdim, q.data_ptr(), H * dim, gate.data_ptr(), H * vdim, 0, kp.data_ptr(), 0,
                                            vp.data_ptr(), 0, pt.data_ptr(), cols, 64, slot.data_ptr(), tp.data_ptr(), n, H, G, dim, vdim,
                                            dim ** -0.5, window, keep, chunk, slopes.data_ptr(), 0, None, sink.data_ptr(), None, 0, 1.0,
                                            None, 0, cabi.DTYPE_CODE[dtype], st))
    for t, p in enumerate(pos):
        j = torch.arange(p + 1, device="cuda")
        seen = torch.ones_like(j, dtype=torch.bool)
        if window:
            seen = (p - j < window) | (j < keep)
        if chunk:
            seen &= j // chunk == p // chunk
        k, v = (x[pt[t].long()].reshape(-1, G, w)[:p + 1].to(F64).repeat_interleave(H // G, 1) for x, w in ((kp, dim), (vp, vdim)))
        s = torch.einsum("hd,nhd->hn", q[t].view(H, dim).to(F64), k) * dim ** -0.5 - slopes.to(F64)[:, None] * (p - j)
        s = torch.cat([s.masked_fill(~seen, -math.inf), sink.to(F64)[:, None]], 1)
        want = torch.einsum("hn,nhd->hd", torch.softmax(s, -1)[:, :-1], v).reshape(-1) * torch.sigmoid(gate[t].to(F64))
        assert _rel(out[t], want) < _tol(dtype, 4e-3)    # one rounding of the result; weights are fp32


def _single_tokens(q, kp, vp, pos, H, G, dim, vdim, scale, head_bias=None, sigmoid=0):
    cabi, L, st = _cabi()
    n, dt = q.shape[0], q.dtype
    cols = kp.shape[0] // n
    pt = torch.arange(n * cols, dtype=torch.int32, device="cuda")
    slot, tp = torch.arange(n, dtype=torch.int32, device="cuda"), torch.tensor(pos, dtype=torch.int32, device="cuda")
    out, ws = torch.zeros(n, H * vdim, dtype=dt, device="cuda"), torch.empty(1 << 20, device="cuda")
    cabi.check(L.pg_attention_ragged_ex(out.data_ptr(), H * vdim, q.data_ptr(), H * dim, None, 0, 0, kp.data_ptr(), vp.data_ptr(),
                                        pt.data_ptr(), cols, 64, slot.data_ptr(), tp.data_ptr(), n, H, G, dim, vdim, scale, 0, 0, None, sigmoid,
                                        None if head_bias is None else head_bias.data_ptr(), 1.0, ws.data_ptr(), ws.numel(),
                                        cabi.DTYPE_CODE[dt], st))
    return out


@pytest.mark.parametrize("dim,vdim,H,G", [(64, 64, 4, 4), (128, 128, 16, 4), (256, 192, 5, 1), (256, 256, 8, 1)])
@pytest.mark.parametrize("lo,hi", [(0, 16), (16, 48), (100, 1000)])
def test_single_tokens_scores_of_minus_infinity(dim, vdim, H, G, lo, hi):
    """Keys [lo, hi) whose scores are -inf weigh nothing, wherever the chunks, warps and clusters cut."""
    g = torch.Generator(device="cuda").manual_seed(dim + lo)
    pos, cols = [47, 63, 200, 1279], 20
    kp, vp = _randn(g, 4 * cols, 64, G * dim, std=1e-20), _randn(g, 4 * cols, 64, G * vdim)
    q = torch.full((4, H * dim), 1e20, dtype=BF, device="cuda")
    kp.view(4, -1, G * dim)[:, lo:hi] = -1e20                    # products of -1e40
    out = _single_tokens(q, kp, vp, pos, H, G, dim, vdim, dim ** -0.5)
    for t, p in enumerate(pos):
        k, v = (x.view(4, -1, G, w)[t, :p + 1].to(F64).repeat_interleave(H // G, 1) for x, w in ((kp, dim), (vp, vdim)))
        s = torch.einsum("hd,nhd->hn", q[t].view(H, dim).to(F64), k) * dim ** -0.5
        s[:, lo:hi] = -math.inf
        want = torch.einsum("hn,nhd->hd", torch.softmax(s, -1), v).reshape(-1)
        assert _rel(out[t], want) < 4e-3                         # one rounding of the result; weights are fp32


@pytest.mark.parametrize("dtype,rel", [(BF, 4e-3), (torch.float16, 6e-4)])
@pytest.mark.parametrize("dim,vdim,H,G", [(64, 64, 4, 4), (128, 128, 16, 4), (256, 192, 5, 1), (256, 256, 8, 1)])
@pytest.mark.parametrize("sigmoid,low", [(0, -15.0), (0, -9.25), (1, -14.0), (1, -17.5), (1, -2.0)])
def test_single_tokens_small_weights(dtype, rel, dim, vdim, H, G, sigmoid, low):
    """Softmax: one key of weight 1 and value 0 beside many of weight exp(low) and value 1.  Sigmoid: nothing but weights of
    sigmoid(low), of which fp16 itself would hold a few bits or none."""
    n, cols, pos = 3, 40, [1, 700, 2559]
    new = lambda f, *s: torch.full(s, f, dtype=dtype, device="cuda")  # noqa: E731
    kp, vp, q = new(0.0, n * cols, 64, G * dim), new(1.0, n * cols, 64, G * vdim), new(0.0, n, H * dim)
    q.view(n, H, dim)[:, :, 0] = 1.0
    if not sigmoid:
        kp.view(n, -1, G, dim)[:, 1:, :, 0] = low
        vp.view(n, -1, G * vdim)[:, 0] = 0.0
    out = _single_tokens(q, kp, vp, pos, H, G, dim, vdim, 1.0, torch.full((H,), low, device="cuda") if sigmoid else None, sigmoid)
    for t, p in enumerate(pos):
        small = p * math.exp(low)
        want = (p + 1) / (1.0 + math.exp(-low)) if sigmoid else small / (1.0 + small)
        # one rounding of the result (below 2^-14 an fp16 result is a multiple of 2^-24), up to 2560 fp32 additions
        assert float((out[t].to(F64) - want).abs().max()) < rel * want + (2.0 ** -25 if dtype == torch.float16 else 0.0)


@pytest.mark.parametrize("dtype", [BF, torch.float16])
@pytest.mark.parametrize("sigmoid", [0, 1])
@pytest.mark.parametrize("dim,vdim,H,G", [(64, 64, 4, 4), (128, 128, 16, 4), (256, 192, 5, 1), (256, 256, 8, 1)])
def test_single_tokens_infinite_values(dtype, sigmoid, dim, vdim, H, G):
    """An infinity in a value row makes its column infinite for the tokens that see the key, and no other column."""
    g = torch.Generator(device="cuda").manual_seed(dim + vdim)
    pos, cols = [0, 20, 300, 1279], 20
    kp, vp, q = (_randn(g, *s, dtype=dtype) for s in ((4 * cols, 64, G * dim), (4 * cols, 64, G * vdim), (4, H * dim)))
    v4 = vp.view(4, -1, G, vdim)
    for t, p in enumerate(pos):
        v4[t, 0, :, 3], v4[t, p // 2, :, 40], v4[t, p, :, 50] = math.inf, -math.inf, math.inf
    out = _single_tokens(q, kp, vp, pos, H, G, dim, vdim, dim ** -0.5, torch.full((H,), -3.0, device="cuda") if sigmoid else None, sigmoid)
    for t, p in enumerate(pos):
        k, v = (x.view(4, -1, G, w)[t, :p + 1].to(F64).repeat_interleave(H // G, 1) for x, w in ((kp, dim), (vp, vdim)))
        s = torch.einsum("hd,nhd->hn", q[t].view(H, dim).to(F64), k) * dim ** -0.5
        w = torch.sigmoid(s - 3.0) if sigmoid else torch.softmax(s, -1)
        o, fine = out[t].view(H, vdim), torch.isfinite(v).all(0).all(0)
        assert bool((o[:, 3] == math.inf).all()) and bool((o[:, 40] == -math.inf).all()) and bool((o[:, 50] == math.inf).all())
        want = torch.einsum("hn,nhd->hd", w, v[:, :, fine])
        assert _rel(o[:, fine], want) < 4e-3      # one rounding of the result; weights are fp32


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("M", [16, 129, 256, 260, 384])
@pytest.mark.parametrize("N,K,epi", [(1152, 4304, "bias_res"), (2048, 2048, "res"), (2560, 2048, "none"), (1160, 1152, "bias_gelu"),
                                     (520, 1096, "f32")])
def test_few_tiles_split_over_clusters(M, N, K, epi, dtype):
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, w = _randn(g, M, K, dtype=dtype), _randn(g, N, K, std=K ** -0.5, dtype=dtype)
    r, b = _randn(g, M, N, dtype=dtype), _randn(g, N, dtype=dtype)
    f32 = epi == "f32"
    out = torch.zeros(M + 1, N, dtype=torch.float32 if f32 else dtype, device="cuda")
    code = {"res": cabi.EPI_RES, "bias_res": cabi.EPI_BIAS_RES, "bias_gelu": cabi.EPI_BIAS_GELU}.get(epi, cabi.EPI_NONE)
    has_b, has_r = epi.startswith("bias"), epi.endswith("res")
    cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), b.data_ptr() if has_b else None, r.data_ptr() if has_r else None, M, N,
                         K, K, K, N, N if has_r else 0, 0, code, 1 if f32 else 0, 2, cabi.DTYPE_CODE[dtype], st))
    want = a.to(F64) @ w.to(F64).T
    if has_b:
        want = want + b.to(F64)
    if epi == "bias_gelu":
        want = _gelu(want)
    if has_r:
        want = want + r.to(F64)
    assert _rel(out[:M], want) < _tol(dtype, 4e-3, epi == "bias_gelu")    # at most three roundings of 2^-9 and the hardware tanh
    assert bool((out[M] == 0).all())


@pytest.mark.parametrize("rows", [1, 2, 3, 1023, 1024, 1025])
@pytest.mark.parametrize("D", [8, 1152, 1288, 2048])
def test_norm_rows(rows, D):
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    x, w, b = _randn(g, rows, D), _randn(g, D), _randn(g, D)
    out = torch.zeros(rows + 1, D, dtype=BF, device="cuda")
    xf = x.to(F64)
    cabi.check(L.pg_rmsnorm(out.data_ptr(), x.data_ptr(), w.data_ptr(), rows, D, 1e-6, cabi.PG_BF16, st))
    want = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6) * (1 + w.to(F64))
    assert _rel(out[:rows], want) < 2.5e-3     # one rounding of the result, statistics in fp32
    cabi.check(L.pg_layernorm(out.data_ptr(), x.data_ptr(), w.data_ptr(), b.data_ptr(), rows, D, 1e-6, cabi.PG_BF16, st))
    want = F.layer_norm(xf, (D,), w.to(F64), b.to(F64), 1e-6)
    assert _rel(out[:rows], want) < 2.5e-3
    assert bool((out[rows] == 0).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("M", [256, 257, 272, 273, 288, 289, 516])
@pytest.mark.parametrize("N,K,kind", [(9480, 136, "geglu"), (9480, 1000, "geglu"), (9472, 136, "swiglu"), (19000, 72, "none"), (18960, 1000, "res"),
                                      (19000, 1000, "f32")])
def test_rows_behind_a_multiple_of_256(M, N, K, kind, dtype):
    """257 to 288 rows: the remainder rides along with the full 256; the row counts next to them; ragged last tiles."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(M + K)
    dual, f32 = kind.endswith("glu"), kind == "f32"
    a, w, r = _randn(g, M, K, dtype=dtype), _randn(g, 2 * N if dual else N, K, std=K ** -0.5, dtype=dtype), _randn(g, M, N, dtype=dtype)
    out = torch.zeros(M + 1, N, dtype=torch.float32 if f32 else dtype, device="cuda")
    code = {"geglu": cabi.EPI_GEGLU, "swiglu": cabi.EPI_SWIGLU, "res": cabi.EPI_RES}.get(kind, cabi.EPI_NONE)
    res = kind == "res"
    cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), None, r.data_ptr() if res else None, M, N, K, K, K, N, N if res else 0, 0,
                         code, 1 if f32 else 0, 2, cabi.DTYPE_CODE[dtype], st))
    z = a.to(F64) @ w.to(F64).T
    want = {"geglu": lambda: _gelu(z[:, :N]) * z[:, N:], "swiglu": lambda: F.silu(z[:, :N]) * z[:, N:], "res": lambda: z + r.to(F64)}.get(kind, lambda: z)()
    tol = _tol(dtype, 5e-3, kind == "geglu")    # up to three roundings of 2^-9 (the fp32 rows hold values rounded to 16 bits) and the tanh
    for rows in (slice(0, 256), slice(256, M))[:1 if M == 256 else 2]:
        assert _rel(out[:M][rows], want[rows]) < tol
    assert bool((out[M] == 0).all())


def test_im2col_rows_at_the_end_of_32_bits():
    """The last patch rows below 2^31: one channel of 2 x 2 pixels is one patch of 2 rows, so the output equals the input."""
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 2 x 8.6 GB beside its comparison")
    cabi, L, st = _cabi()
    B = 2 ** 30 - 8                                              # 2^31 - 16 patch rows
    x = torch.empty(4 * B, dtype=torch.int16, device="cuda").random_(0, 2 ** 15 - 1)
    out = torch.zeros_like(x)
    cabi.check(L.pg_im2col(out.data_ptr(), x.data_ptr(), B, 1, 2, 2, 2, 4, cabi.PG_BF16, st))
    assert all(torch.equal(a, b) for a, b in zip(out.split(1 << 30), x.split(1 << 30)))


@pytest.mark.parametrize("M", [8, 40, 100, 260])
@pytest.mark.parametrize("N,K,epi", [(2048, 2048, "none"), (1152, 4304, "res"), (1024, 1024, "bias")])
def test_weights_written_by_the_launch_before(M, N, K, epi):
    """W = U V^T comes from a pg_gemm right in front of the one that multiplies with it, over the rest of another W."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    u, v, a, r, b = _randn(g, N, 512, std=512 ** -0.5), _randn(g, K, 512), _randn(g, M, K, std=K ** -0.5), _randn(g, M, N), _randn(g, N)
    w, out = torch.empty(N, K, dtype=BF, device="cuda"), torch.empty(M, N, dtype=BF, device="cuda")
    code = {"res": cabi.EPI_RES, "bias": cabi.EPI_BIAS, "none": cabi.EPI_NONE}[epi]
    z = a.to(F64) @ (u.to(F64) @ v.to(F64).T).to(BF).to(F64).T
    want = z + (r.to(F64) if epi == "res" else b.to(F64) if epi == "bias" else 0.0)
    for _ in range(20):
        w.fill_(1e4)
        cabi.check(L.pg_gemm(w.data_ptr(), u.data_ptr(), v.data_ptr(), None, None, N, K, 512, 512, 512, K, 0, 0, 0, 0, 0, cabi.PG_BF16, st))
        cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), b.data_ptr(), r.data_ptr(), M, N, K, K, K, N, N, 0, code, 0, 0,
                             cabi.PG_BF16, st))
        # W's elements round either way at their ties with the exact product (2^-9 of a few), the result is rounded once or twice
        assert _rel(out, want) < 6e-3


@pytest.mark.parametrize("sigmoid", [0, 1])
def test_window_gates_and_weights_near_the_smallest_number(sigmoid):
    """sigmoid(-87.5) is 1e-38: times values of 1e38 that is an ordinary number, for the gate and for a sigmoid weight."""
    cabi, L, st = _cabi()
    n, H, d, at = 70, 2, 64, -87.5
    new = lambda f, *s: torch.full(s, f, dtype=BF, device="cuda")  # noqa: E731
    q, kp, vp, gate = new(0.0, n, H * d), new(0.0, 2, 64, H * d), new(1e38, 2, 64, H * d), new(at, n, H * d)
    pt = torch.tensor([[1, 0]], dtype=torch.int32, device="cuda")
    tiles = torch.tensor([[0, n, 0, 0]], dtype=torch.int32, device="cuda")
    bias, err = torch.full((H,), at, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(n, H * d, dtype=BF, device="cuda")
    cabi.check(L.pg_attention_ragged_tc_ex(out.data_ptr(), H * d, q.data_ptr(), H * d, None if sigmoid else gate.data_ptr(), H * d, 0,
                                           kp.data_ptr(), vp.data_ptr(), 128, pt.data_ptr(), 2, 64, tiles.data_ptr(), 1, n, H, H, d, d,
                                           1.0, 1, 0, None, sigmoid, bias.data_ptr() if sigmoid else None, 1.0, err.data_ptr(),
                                           cabi.PG_BF16, st))
    want = float(vp[0, 0, 0]) * math.exp(at)
    assert int(err) == 0
    # exp(87.5) as 2^x: the exponent's rounding, 2^-18 of 126, is 3e-4 of the result; a weight of 1e-38 keeps 8 bits or, if the
    # type's subnormal numbers are meant, 7; one rounding of the result
    assert float((out.to(F64) - want).abs().max()) < 1.2e-2 * want


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("dim,vdim,H,G", [(64, 64, 2, 1), (64, 192, 4, 2), (128, 144, 2, 1), (72, 136, 2, 2), (256, 192, 2, 1), (256, 256, 2, 1)])
@pytest.mark.parametrize("window", [0, 65, 200])
def test_window_prompts(dim, vdim, H, G, window, dtype):
    """Prompt tiles of 128 and 72 rows behind 30 cached tokens, at value widths on both sides of what 256 columns of TMEM hold."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(dim + vdim)
    past, T, cols = 30, 200, 4
    kp, vp = _randn(g, cols + 1, 64, G * dim, dtype=dtype), _randn(g, cols + 1, 64, G * vdim, dtype=dtype)
    q, gate = _randn(g, T, H * dim, dtype=dtype), _randn(g, T, H * vdim, dtype=dtype)
    pt = torch.randperm(cols + 1, device="cuda", generator=g)[:cols].to(torch.int32).view(1, cols)
    tiles = torch.tensor([[0, 128, 0, past], [128, 72, 0, past + 128]], dtype=torch.int32, device="cuda")
    slopes, err = torch.rand(H, device="cuda", generator=g) * 0.2, torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(T + 1, H * vdim, dtype=dtype, device="cuda")
    cabi.check(L.pg_attention_ragged_tc_capped(out.data_ptr(), H * vdim, q.data_ptr(), H * dim, gate.data_ptr(), H * vdim, 0, kp.data_ptr(), 0,
                                               vp.data_ptr(), 0, (cols + 1) * 64, pt.data_ptr(), cols, 64, tiles.data_ptr(), 2, T, H, G, dim,
                                               vdim, dim ** -0.5, window, 0, 0, slopes.data_ptr(), 0, None, None, 0.0, 0.0, 0, None, 0, 1.0,
                                               err.data_ptr(), cabi.DTYPE_CODE[dtype], st))
    i, j = torch.arange(T, device="cuda")[:, None] + past, torch.arange(past + T, device="cuda")[None]
    seen = (j <= i) & ((i - j < window) if window else (j >= 0))
    k, v = (x[pt[0].long()].reshape(-1, G, w)[:past + T].to(F64).repeat_interleave(H // G, 1) for x, w in ((kp, dim), (vp, vdim)))
    s = torch.einsum("qhd,nhd->hqn", q.view(T, H, dim).to(F64), k) * dim ** -0.5 - slopes.to(F64)[:, None, None] * (i - j)
    want = torch.einsum("hqn,nhd->qhd", torch.softmax(s.masked_fill(~seen, -math.inf), -1), v).reshape(T, -1) * torch.sigmoid(gate.to(F64))
    assert int(err) == 0
    assert _rel(out[:T], want) < _tol(dtype, 5e-3)      # weights and result are rounded once each
    assert bool((out[T] == 0).all())


def _scan_columns(seqs, heads, dim, vdim):
    """Value columns per thread: by the warps of the one-column form, with 4, 8 or 16 lanes a column."""
    warps = seqs * heads * vdim * (4 if dim <= 32 else 8 if dim <= 128 else 16) / 32
    return 4 if warps >= 1536 else 2 if warps >= 768 else 1


@pytest.mark.parametrize("dim,vdim", [(20, 128), (32, 136), (64, 130), (100, 131), (128, 256), (200, 132), (256, 128)])
@pytest.mark.parametrize("per_channel", [0, 1])
def test_linear_scan_alone_and_in_a_batch(dim, vdim, per_channel):
    """One or two value columns per thread for a sequence alone, four for the batch: the same sums in the same order, to the bit."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(dim + vdim)
    H, lens = 16, [70, 1, 3, 16, 33, 8]
    S, T, dp, vp = len(lens), sum(lens), -(-dim // 4) * 4, -(-vdim // 4) * 4
    nq = 3 if per_channel else 2
    rec = torch.zeros(T, H, nq * dp + vp, device="cuda")
    q, k, v = (torch.randn(T, H, w, device="cuda", generator=g) for w in (dim, dim, vdim))
    decay = torch.rand(T, H, dim, device="cuda", generator=g) if per_channel else torch.linspace(0.5, 0.99, H, device="cuda")
    rec[:, :, :dim], rec[:, :, dp:dp + dim], rec[:, :, nq * dp:nq * dp + vdim] = q, k, v
    if per_channel:
        rec[:, :, 2 * dp:2 * dp + dim] = decay
    start = torch.randn(S, H, dim, vdim, device="cuda", generator=g)
    first = [sum(lens[:b]) for b in range(S)]

    def scan(segs, state):
        out = torch.full((T, H, vdim), 7.0, device="cuda")
        sg = torch.tensor(segs, dtype=torch.int32, device="cuda")
        if per_channel:
            cabi.check(L.pg_gla_attention(out.data_ptr(), state.data_ptr(), rec.data_ptr(), sg.data_ptr(), len(segs), H, dim, vdim, st))
        else:
            cabi.check(L.pg_lightning_attention(out.data_ptr(), state.data_ptr(), rec.data_ptr(), decay.data_ptr(), sg.data_ptr(), len(segs), H,
                                                dim, vdim, st))
        torch.cuda.synchronize()
        return out, state

    out, state = scan([[b, first[b], lens[b]] for b in range(S)], start.clone())
    assert _scan_columns(S, H, dim, vdim) == 4 > _scan_columns(1, H, dim, vdim)
    for b in range(S):
        rows = slice(first[b], first[b] + lens[b])
        o1, s1 = scan([[b, first[b], lens[b]]], start.clone())
        assert torch.equal(o1[rows], out[rows]) and torch.equal(s1[b], state[b])
        x, want = start[b].to(F64), []
        for t in range(rows.start, rows.stop):
            a = decay[t].to(F64)[:, :, None] if per_channel else decay.to(F64)[:, None, None]
            x = a * x + k[t].to(F64)[:, :, None] * v[t].to(F64)[:, None, :]
            want.append(torch.einsum("hd,hdv->hv", q[t].to(F64), x))
        assert _rel(out[rows], torch.stack(want)) < 2e-6 and _rel(state[b], x) < 2e-6   # fp32 sums of up to 256 products


@pytest.mark.parametrize("kind", ["head", "token", "channel"])
@pytest.mark.parametrize("H,dim,vdim,lens", [(2, 32, 20, [1, 2, 3, 4, 5, 31, 32, 33, 300]), (3, 128, 36, [7, 64, 129]),
                                             (2, 256, 130, [3, 70]), (16, 128, 128, [1, 3, 4, 2, 9] * 13)])
def test_linear_scan_steps_of_four(kind, H, dim, vdim, lens):
    """Whole and partial steps of four tokens, the ring of prepared steps and its second round, short segments and many of
    them, a decay of 0, of 1 and just below it, and a later token's infinity."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(dim + vdim)
    S, T, dp, vp = len(lens), sum(lens), -(-dim // 4) * 4, -(-vdim // 4) * 4
    nq, tail = (3, 0) if kind == "channel" else (2, 4 if kind == "token" else 0)
    q, k, v = (torch.randn(T, H, w, device="cuda", generator=g) for w in (dim, dim, vdim))
    by_head = torch.linspace(0.99, 0.999, H, device="cuda")
    by_head[0] = 0.0
    a = {"head": lambda: by_head.view(1, H, 1).expand(T, H, dim), "channel": lambda: torch.rand(T, H, dim, device="cuda", generator=g) ** 0.1,
         "token": lambda: (torch.rand(T, H, 1, device="cuda", generator=g) ** 0.1).expand(T, H, dim)}[kind]().clone()
    if kind != "head":
        a[1:3] = 1.0
    rec = torch.zeros(T, H, nq * dp + vp + tail, device="cuda")
    rec[:, :, :dim], rec[:, :, dp:dp + dim], rec[:, :, nq * dp:nq * dp + vdim] = q, k, v
    if kind == "channel":
        rec[:, :, 2 * dp:2 * dp + dim] = a
    if kind == "token":
        rec[:, :, nq * dp + vp] = a[:, :, 0]
    skip = torch.randn(H, device="cuda", generator=g) if kind == "token" else None
    first = [sum(lens[:b]) for b in range(S)]
    segs = torch.tensor([[b, first[b], lens[b]] for b in range(S)] + [[0, 0, 0]], dtype=torch.int32, device="cuda")
    start = torch.randn(S, H, dim, vdim, device="cuda", generator=g)

    def scan(rec):
        out, state = torch.full((T, H, vdim), 7.0, device="cuda"), start.clone()
        if kind == "channel":
            cabi.check(L.pg_gla_attention(out.data_ptr(), state.data_ptr(), rec.data_ptr(), segs.data_ptr(), S + 1, H, dim, vdim, st))
        else:
            cabi.check(L.pg_lightning_attention_ex(out.data_ptr(), state.data_ptr(), rec.data_ptr(), by_head.data_ptr() if kind == "head" else None,
                                                   None if skip is None else skip.data_ptr(), segs.data_ptr(), S + 1, H, dim, vdim, st))
        torch.cuda.synchronize()
        return out, state

    out, state = scan(rec)
    want, end = torch.empty(T, H, vdim, dtype=F64, device="cuda"), start.to(F64)
    for b in range(S):
        x = end[b]
        for t in range(first[b], first[b] + lens[b]):
            x = a[t].to(F64)[:, :, None] * x + k[t].to(F64)[:, :, None] * v[t].to(F64)[:, None, :]
            want[t] = torch.einsum("hd,hdv->hv", q[t].to(F64), x) + (0 if skip is None else skip.to(F64)[:, None] * v[t].to(F64))
        end[b] = x
    # a product of dim terms and a state of some hundred: a few roundings of 2^-24 each, in quadrature
    assert _rel(out, want) < 1e-6 and _rel(state, end) < 1e-6
    if lens[0] > 1 or lens[1] > 2:
        at = first[-1] + lens[-1] - 1                     # the last token of the last segment: nothing before it may notice
        bad = rec.clone()
        bad[at, :, nq * dp:nq * dp + vdim] = float("inf")
        out2, state2 = scan(bad)
        keep = torch.arange(T, device="cuda") != at
        assert torch.equal(out2[keep], out[keep]) and not bool(torch.isfinite(out2[at]).any())
        assert torch.equal(state2[:-1], state[:-1]) and not bool(torch.isfinite(state2[-1, :, :dim]).any())


@pytest.mark.parametrize("kind", ["head", "token", "channel"])
@pytest.mark.parametrize("dim", [24, 60, 100, 200])
@pytest.mark.parametrize("columns,vdim", [(1, 131), (2, 131), (2, 132), (4, 130), (4, 132)])
def test_linear_scan_value_columns(columns, vdim, dim, kind):
    """Every form (value columns per thread, key width, kind of decay), whole and partial groups of columns: to the bit what a
    sequence gives alone, and a float64 recurrence."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(dim + vdim + columns)
    H, n, dp, vp = 8, 10, -(-dim // 4) * 4, -(-vdim // 4) * 4
    S = columns * (4 if dim <= 32 else 2 if dim <= 128 else 1)
    assert _scan_columns(S, H, dim, vdim) == columns and _scan_columns(1, H, dim, vdim) == 1
    nq, tail = (3, 0) if kind == "channel" else (2, 4 if kind == "token" else 0)
    q, k, v = (torch.randn(S * n, H, w, device="cuda", generator=g) for w in (dim, dim, vdim))
    by_head = torch.linspace(0.5, 0.99, H, device="cuda")
    wide = {"head": 1, "token": 1, "channel": dim}[kind]
    a = by_head.view(1, H, 1).expand(S * n, H, 1) if kind == "head" else torch.rand(S * n, H, wide, device="cuda", generator=g)
    rec = torch.zeros(S * n, H, nq * dp + vp + tail, device="cuda")
    rec[:, :, :dim], rec[:, :, dp:dp + dim], rec[:, :, nq * dp:nq * dp + vdim] = q, k, v
    if kind == "channel":
        rec[:, :, 2 * dp:2 * dp + dim] = a
    if kind == "token":
        rec[:, :, nq * dp + vp] = a[:, :, 0]
    start = torch.randn(S, H, dim, vdim, device="cuda", generator=g)

    def scan(seqs):
        out, state = torch.full((S * n, H, vdim), 7.0, device="cuda"), start.clone()
        segs = torch.tensor([[b, b * n, n] for b in seqs], dtype=torch.int32, device="cuda")
        cabi.check(L.pg_linear_scan(out.data_ptr(), state.data_ptr(), rec.data_ptr(), by_head.data_ptr() if kind == "head" else None, None,
                                    1 if kind == "channel" else 0, segs.data_ptr(), len(seqs), H, dim, vdim, 0, None, st))
        torch.cuda.synchronize()
        return out, state

    out, state = scan(list(range(S)))
    x, want = start.to(F64), []
    q64, k64, v64, a64 = (z.to(F64).view(S, n, H, -1) for z in (q, k, v, a.contiguous()))
    for t in range(n):
        x = a64[:, t, :, :, None] * x + k64[:, t, :, :, None] * v64[:, t, :, None, :]
        want.append(torch.einsum("shd,shdv->shv", q64[:, t], x))
    # a product of dim terms and a state of some units: a few roundings of 2^-24 each, in quadrature
    assert _rel(out, torch.stack(want, 1).view(S * n, H, vdim)) < 1e-6 and _rel(state, x) < 1e-6
    for b in (0, S - 1):
        o1, s1 = scan([b])
        assert torch.equal(o1[b * n:(b + 1) * n], out[b * n:(b + 1) * n]) and torch.equal(s1[b], state[b])


@pytest.mark.parametrize("per_channel", [0, 1])
@pytest.mark.parametrize("H,dim,vdim,lens", [(2, 32, 20, [40, 3, 9]), (3, 128, 36, [100, 4, 1]), (16, 64, 128, [5, 2, 70, 33])])
def test_linear_scan_waits_that_run_out(H, dim, vdim, lens, per_channel):
    """Waits that count as run out: the flag is set, outputs and states of the segments that wait are NaN, shorter segments have
    their results; nothing is written outside the segments, and the next call is whole again."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(dim + vdim)
    S, T, dp, vp, nq = len(lens), sum(lens), dim, -(-vdim // 4) * 4, 3 if per_channel else 2
    rec = torch.rand(T, H, nq * dp + vp, device="cuda", generator=g) * 0.9
    decay = None if per_channel else torch.linspace(0.5, 0.99, H, device="cuda")
    first = [sum(lens[:b]) for b in range(S)]
    segs = torch.tensor([[b, first[b], lens[b]] for b in range(S)], dtype=torch.int32, device="cuda")
    start = torch.randn(S + 1, H, dim, vdim, device="cuda", generator=g)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def scan(no_wait, flag):
        out, state = torch.full((T + 1, H, vdim), 7.0, device="cuda"), start.clone()
        cabi.check(L.pg_linear_scan(out.data_ptr(), state.data_ptr(), rec.data_ptr(), cabi.ptr(decay), None, per_channel, segs.data_ptr(), S, H,
                                    dim, vdim, no_wait, cabi.ptr(flag), st))
        torch.cuda.synchronize()
        return out, state

    out, state = scan(0, err)
    assert int(err) == 0 and bool(torch.isfinite(out).all()) and bool(torch.isfinite(state).all())
    for flag in (None, err):
        lost, gone = scan(1, flag)
        for b in range(S):
            rows = slice(first[b], first[b] + lens[b])
            if lens[b] < 4:
                assert torch.equal(lost[rows], out[rows]) and torch.equal(gone[b], state[b])
            else:
                assert bool(torch.isnan(lost[rows]).all()) and bool(torch.isnan(gone[b]).all())
        assert bool((lost[T] == 7).all()) and torch.equal(gone[S], start[S])
    assert int(err) == 2
    again, state2 = scan(0, None)
    assert torch.equal(again, out) and torch.equal(state2, state)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(4, 8, 8), (7, 1184, 72), (8, 1192, 1024), (9, 2368, 1032), (16, 2376, 2048), (17, 2048, 2048), (32, 1000, 2040),
                                   (12, 9472, 520), (5, 2048, 16384), (16, 2048, 8200), (1, 2367, 72), (2, 2048, 16384), (3, 1001, 4104),
                                   (1, 2367, 2056), (2, 504, 648), (2, 776, 8200), (3, 8, 1032), (3, 1784, 8192), (7, 2376, 512), (16, 9472, 4096)])
def test_streamed_rows(M, N, K, dtype):
    """Every SM's share of weight rows: fewer rows than CTAs, shares of 8, 9, 16 and 17 rows (a second group), four groups, columns that
    end inside a lane's step and behind a chunk; one to three rows of a decode step, features that are no multiple of 8."""
    cabi, L, st = _cabi()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    pad = 8 if M > 3 else 0
    a, w = _randn(g, M, K + pad, dtype=dtype), _randn(g, N, K + pad, std=K ** -0.5, dtype=dtype)
    b, r = _randn(g, N, dtype=dtype), _randn(g, M, N + pad, dtype=dtype)
    y = a[:, :K].to(F64) @ w[:, :K].to(F64).T
    y_b, res = y + b.to(F64), r[:, :N].to(F64)
    want = {cabi.EPI_NONE: y, cabi.EPI_RES: y + res, cabi.EPI_BIAS: y_b, cabi.EPI_BIAS_RES: y_b + res,
            cabi.EPI_BIAS_GELU: torch.nn.functional.gelu(y_b, approximate="tanh")}
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for epi, ref in want.items():
        for f32 in (0, 1) if M > 3 else (0,):
            out = torch.full((M + 1, N + pad), 7.0, dtype=torch.float32 if f32 else dtype, device="cuda")
            if M > 3:
                cabi.check(L.pg_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), b.data_ptr(), r.data_ptr(), M, N, K, K + pad, K + pad, N + pad,
                                     N + pad, 0, epi, f32, 2 | cabi.GEMM_W_PARAM, cabi.DTYPE_CODE[dtype], st))
            elif epi in (cabi.EPI_NONE, cabi.EPI_RES):
                cabi.check(L.pg_gemv_res(out.data_ptr(), a.data_ptr(), w.data_ptr(), r.data_ptr() if epi == cabi.EPI_RES else None, M, N, K, None,
                                         cabi.DTYPE_CODE[dtype], st))
            else:
                continue
            # up to three roundings (product, activation, sum) of half a step of the type each, and the fast tanh's 2^-11
            assert _rel(out[:M, :N], ref) < 1.5 * eps + 2.0 ** -11 and float((out[:M, :N].to(F64) - ref).abs().max()) < 4 * eps * float(ref.abs().max())
            assert bool((out[M] == 7).all()) and bool((out[:, N:] == 7).all())
