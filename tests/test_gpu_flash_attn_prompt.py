"""The fast prompt-attention kernel (csrc/flash_attn_prompt.cu) where it can go wrong: edges of its 128-row blocks and 128-position tiles, positions
over one to eight CTAs, mask rows on and off 16-byte boundaries, tiles that are clear, hidden or mixed, running maxima that grow (-m gpu).

Tolerance, per output row relative to the row's largest magnitude, against float64 with q rounded to f16 (as the operation rounds it): the weights
of 64 and more rows are rounded to f16 before the second product and in the sum alike, 2^-11 of each weight, which over a row gives at most
2 * 2^-11 = 9.8e-4 of the largest |v|; 1e-3 as asked of F16-KV attention."""
import ctypes as C

import numpy as np
import pytest

import b200
from test_gpu_flash_attn import synth_case
from test_gpu_flash_attn_fast import ref64, row_rel

pytestmark = pytest.mark.gpu
TOL = 1e-3


@pytest.fixture(scope="module")
def dev():
    mod = b200.load()
    assert mod.device_count() > 0
    mod.set_device(0)
    return mod


def check(dev, q, k, v, mask, scale, got=None, coarse=()):
    """coarse: rows whose scores carry a bias of -65504 everywhere: in log2 units an F32 step there is 2^-7, so that every weight is off by up to
    2^-8 ln 2 = 2.7e-3 of itself; 1e-2 for an output that is smaller than the values it is made of"""
    if got is None:
        got = dev.flash_attn(q, dev.KvCacheView(k, v), mask, scale, mode=1)
    assert dev.kernel_error() == 0
    live = np.ones(q.shape[1], bool) if mask is None else (mask != 0xFC00).any(axis=1)
    assert not got[~live].any()
    with np.errstate(invalid="ignore"):
        want = ref64(q.astype(np.float16).astype(np.float32), k, v, mask, scale)
    fine = live.copy()
    fine[list(coarse)] = False
    assert row_rel(got[fine], want[fine]) <= TOL
    for t in coarse:
        assert row_rel(got[t], want[t]) <= 1e-2


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H,Hkv,T", [(4, 4, 64), (4, 2, 64), (8, 2, 33), (6, 2, 43), (16, 1, 65), (3, 1, 2)], ids=str)
@pytest.mark.parametrize("n_kv", [127, 128, 129, 256, 777, 2050])
def test_edges(dev, D, H, Hkv, T, n_kv):
    """row blocks that are full, ragged, or begin inside a token; caches of less than a tile, whole tiles, a position more; the mask's rows start on
    2-byte, 4-byte and 16-byte boundaries"""
    q, k, v, mask = synth_case(H, Hkv, D, T, n_kv, seed=D + H * T + n_kv)
    check(dev, q, k, v, mask, D ** -0.5)
    if T >= 64:
        check(dev, q, k, v, None, D ** -0.5)


@pytest.mark.parametrize("n_kv", [1, 5])
def test_a_cache_of_a_few_positions(dev, n_kv):
    q, k, v, _ = synth_case(8, 2, 128, 64, n_kv, seed=n_kv, causal=False)
    check(dev, q, k, v, None, 0.09)


@pytest.mark.parametrize("n_kv", [1100, 1104])
def test_masks_of_any_values(dev, n_kv):
    """finite biases, the type's lowest value, hidden and clear tiles, rows that see nothing or only the last position"""
    rng = np.random.default_rng(n_kv)
    H, Hkv, D, T = 8, 4, 128, 70
    q, k, v, _ = synth_case(H, Hkv, D, T, n_kv, seed=3, causal=False)
    m = (rng.standard_normal((T, n_kv)) * 2).astype(np.float16)
    m[:, 128:384] = 0.0
    m[:, 512:768] = -np.inf
    m[10:20, :] = np.float16(-65504.0)
    m[10:20, 1000] = 0.0
    m[21, :] = np.float16(-65504.0)
    m[30:34, :] = -np.inf
    m[40:50, :] = -np.inf
    m[40:50, n_kv - 1] = 0.0
    check(dev, q, k, v, m.view(np.uint16), D ** -0.5, coarse=[21])


@pytest.mark.parametrize("D", [64, 128])
def test_maxima_that_grow_along_the_cache(dev, D):
    """scores that rise by far more than 2^8 from tile to tile, and fall for other rows: outputs are rescaled often, or never"""
    H, Hkv, T, n_kv = 4, 2, 100, 1500
    q, k, v, mask = synth_case(H, Hkv, D, T, n_kv, seed=D, causal=True)
    ramp = (np.arange(n_kv) / 100.0).astype(np.float32)
    kf = k.view(np.float16).astype(np.float32)
    kf[:, :, 0] = ramp
    q[:, ::2, 0] = 8.0 * D ** 0.5
    q[:, 1::2, 0] = -8.0 * D ** 0.5
    check(dev, q, kf.astype(np.float16).view(np.uint16), v, mask, D ** -0.5)


def test_a_negative_scale(dev):
    q, k, v, mask = synth_case(8, 2, 64, 80, 900, seed=8)
    check(dev, q, k, v, mask, -0.125)


def test_strided_views(dev):
    """q token-major, the cache head-major with gaps, mask rows with a stride of their own and an odd start"""
    H, Hkv, D, T, n_kv = 8, 2, 128, 66, 530
    q, k, v, mask = synth_case(H, Hkv, D, T, n_kv, seed=21)
    pad = 8
    kc = np.full((Hkv, n_kv + 3, D + pad), 0x7E00, np.uint16)   # NaN between the rows
    vc = kc.copy()
    kc[:, :n_kv, :D], vc[:, :n_kv, :D] = k, v
    mc = np.zeros((T, n_kv + 7), np.uint16)
    mc[:, 1:1 + n_kv] = mask
    dq, dk, dv, dm = (dev.device_array(np.ascontiguousarray(x)) for x in (np.transpose(q, (1, 0, 2)), kc, vc, mc))
    dst = dev.DeviceBuffer(4 * T * H * D)
    a = dev.FlashAttnArgs()
    a.dk, a.dv, a.n_tok, a.n_head, a.n_head_kv, a.n_kv = D, D, T, H, Hkv, n_kv
    a.q, a.q_nb1, a.q_nb2 = dq.ptr, H * D * 4, D * 4
    a.k, a.k_nb1, a.k_nb2 = dk.ptr, (D + pad) * 2, (n_kv + 3) * (D + pad) * 2
    a.v, a.v_nb1, a.v_nb2 = dv.ptr, (D + pad) * 2, (n_kv + 3) * (D + pad) * 2
    a.mask, a.mask_nb1 = dm.ptr + 2, (n_kv + 7) * 2
    a.scale, a.dst, a.mode = D ** -0.5, dst.ptr, 1
    dev.check(dev.lib.b200_flash_attn_ext(C.byref(a), None), "flash_attn_ext")
    check(dev, q, k, v, mask, D ** -0.5, dst.download(np.float32, T * H * D).reshape(T, H, D))


def test_few_rows_over_a_long_cache(dev):
    """16 rows over more than 8192 positions: the same function whichever kernel takes them"""
    for n_kv in (8704, 8705):
        q, k, v, mask = synth_case(8, 2, 128, 16, n_kv, seed=n_kv)
        check(dev, q, k, v, mask, 128 ** -0.5)


@pytest.mark.parametrize("H,Hkv,n_kv", [(6, 2, 300), (5, 1, 640), (8, 2, 301), (7, 1, 1023)], ids=str)
def test_few_rows_that_the_decode_kernel_refuses(dev, H, Hkv, n_kv):
    """groups of heads that do not divide 16, mask rows off 4 bytes: under mode 1 the kernel that keeps q and the weights in F32 (1e-5 of float64 with q as
    it is, where q rounded to f16 alone is 2^-11 off), under the fast policy the prompt kernel (1e-5 with q rounded, where the exact kernels' f16 sums are
    1e-3 and more away), whatever a cell holds that nobody sees"""
    T, D = 5, 128
    q, k, v, _ = synth_case(H, Hkv, D, T, n_kv, seed=H + n_kv, causal=False)
    m = np.zeros((T, n_kv), np.float16)
    m[:, 40:44] = -np.inf
    for t in range(T):
        m[t, n_kv - T + t + 1:] = -np.inf
    mask = m.view(np.uint16)
    want = ref64(q, k, v, mask, D ** -0.5)
    want16 = ref64(q16(q), k, v, mask, D ** -0.5)
    got = dev.flash_attn(q, dev.KvCacheView(k, v), mask, D ** -0.5, mode=1)
    assert row_rel(got, want) <= 1e-5
    k, v = k.copy(), v.copy()
    k[:, 41], v[:, 42] = 0x7E00, 0x7C00
    dev.set_numerics(dev.FAST)
    try:
        got = dev.flash_attn(q, dev.KvCacheView(k, v), mask, D ** -0.5)
    finally:
        dev.set_numerics(dev.EXACT)
    assert norm_rel(got, want16) <= 1e-5


def plain(q, k, v, mask, scale):
    """float64, a row at a time over the positions it sees; a score of NaN or +Inf makes the row NaN"""
    H, T, D = q.shape
    G = H // k.shape[0]
    kf, vf = k.view(np.float16).astype(np.float64), v.view(np.float16).astype(np.float64)
    out = np.zeros((T, H, D))
    for h in range(H):
        for t in range(T):
            see = np.arange(k.shape[1]) if mask is None else np.flatnonzero(mask[t] != 0xFC00)
            if len(see) == 0:
                continue
            s = kf[h // G, see] @ q[h, t].astype(np.float16).astype(np.float64) * scale
            if mask is not None:
                s = s + mask[t, see].view(np.float16).astype(np.float64)
            if not (s < np.inf).all():
                out[t, h] = np.nan
                continue
            p = np.exp(s - s.max())
            out[t, h] = (p / p.sum()) @ vf[h // G, see]
    return out


NOT_FINITE = [(8, 2, 64, 256, True), (8, 2, 40, 2056, True), (8, 2, 16, 1032, True), (4, 4, 130, 777, True), (6, 2, 70, 333, True), (8, 4, 96, 640, False)]


@pytest.mark.parametrize("D,H,Hkv,T,n_kv,causal", [(D, *c) for D in (64, 128) for c in NOT_FINITE], ids=str)
def test_values_that_are_not_finite(dev, D, H, Hkv, T, n_kv, causal):
    """A NaN in a query makes its row NaN and no other; NaN and Inf in cells reach the rows that see them and no other, wherever the tiles end: hidden
    from some rows of a tile, from a whole softmax group's tiles, from all rows of a cluster's CTA.  Rows that meet nothing of it keep their bits."""
    scale = D ** -0.5
    q, k, v, mask = synth_case(H, Hkv, D, T, n_kv, seed=D + T, causal=causal)
    if mask is not None:
        mask = mask.copy()
        mask[:, 130:140] = 0xFC00        # cells that nobody sees, inside a tile that all see
        mask[5, :] = 0xFC00
    clean = dev.flash_attn(q, dev.KvCacheView(k, v), mask, scale, mode=1)
    q, k, v = q.copy(), k.copy(), v.copy()
    q[1, 7, 3] = np.nan                  # one head of one token
    q[:, 5, 0] = np.nan                  # a token that sees nothing under the mask
    if mask is not None:
        k[:, 131], v[:, 132], v[:, 133, 1] = 0x7E00, 0x7E00, 0xFC00
    v[0, n_kv - 3, 2] = 0x7C00           # Inf in one channel of a late position: hidden from most rows of a causal batch
    k[Hkv - 1, n_kv - 9, 4] = 0x7E00     # a NaN key
    got = dev.flash_attn(q, dev.KvCacheView(k, v), mask, scale, mode=1)
    assert dev.kernel_error() == 0
    with np.errstate(all="ignore"):
        want = plain(q, k, v, mask, scale)
    assert (np.isnan(got) == np.isnan(want)).all() and (np.isinf(got) == np.isinf(want)).all()
    fine = np.isfinite(want).all(axis=2)
    assert fine.any() and not fine.all()
    assert row_rel(got[fine], want[fine]) <= TOL
    if mask is None:
        untouched = fine.copy()
        untouched[:, H - H // Hkv:] = False
        assert np.array_equal(got[untouched].view(np.uint32), clean[untouched].view(np.uint32))


def test_a_softmax_group_and_a_cta_that_see_nothing_but_nan(dev):
    """keys of tiles 1, 3, .. are NaN (one of two groups of softmax warps; with more tiles than row blocks, whole CTAs of a cluster): no row is finite"""
    for n_kv, T in ((256, 64), (2048, 64), (2048, 300)):
        q, k, v, _ = synth_case(4, 2, 128, T, n_kv, seed=n_kv + T, causal=False)
        k = k.copy()
        for t in range(1, n_kv // 128, 2):
            k[:, 128 * t:128 * (t + 1)] = 0x7E00
        got = dev.flash_attn(q, dev.KvCacheView(k, v), None, 0.09, mode=1)
        assert np.isnan(got).all()


def q16(q):
    return q.astype(np.float16).astype(np.float32)


def norm_rel(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("wide", [1.0, 3.0])
@pytest.mark.parametrize("T,n_kv", [(64, 4096), (300, 1500)])
def test_weights_of_prompts_lose_no_more_than_under_running_maxima(dev, T, n_kv, wide, D):
    """the limit is the distance that rounding each weight to f16 under the running maximum of 64-position tiles alone makes, and a twentieth"""
    H, Hkv = 8, 4
    q, k, v, mask = synth_case(H, Hkv, D, T, n_kv, seed=T + D)
    q, scale = q * wide / q.std(), D ** -0.5 / k.view(np.float16).astype(np.float32).std()
    want = ref64(q16(q), k, v, mask, scale)
    kf, vf, m = k.view(np.float16).astype(np.float64), v.view(np.float16).astype(np.float64), mask.view(np.float16).astype(np.float64)
    rounded = np.empty_like(want)
    for h in range(H):
        s = q16(q)[h].astype(np.float64) @ kf[h // 2].T * scale + m
        top = np.stack([s[:, :64 * (t // 64 + 1)].max(axis=1) for t in range(0, n_kv, 64)], axis=1).repeat(64, axis=1)[:, :n_kv]
        w = np.exp(s - top).astype(np.float16) * np.exp(top - s.max(axis=1, keepdims=True))
        rounded[:, h] = (w / w.sum(axis=1, keepdims=True)) @ vf[h // 2]
    got = dev.flash_attn(q, dev.KvCacheView(k, v), mask, scale, mode=1)
    assert norm_rel(got, want) <= 1.05 * norm_rel(rounded, want)


@pytest.mark.parametrize("wide", [1.0, 3.0])
@pytest.mark.parametrize("T,n_kv", [(12, 1024), (16, 2049), (63, 4096)])
def test_weights_of_a_few_rows_are_two_parts(dev, T, n_kv, wide):
    """weights to 2^-22 of themselves and 2^-25 of the largest, sums of up to 4096 F32 terms: 1e-5, where f16 weights are 2e-4 away (2049 positions: mask
    rows off 4 bytes, the kernel in F32)"""
    D = 128
    q, k, v, mask = synth_case(8, 2, D, T, n_kv, seed=T + D)
    q, scale = q * wide / q.std(), D ** -0.5 / k.view(np.float16).astype(np.float32).std()
    got = dev.flash_attn(q, dev.KvCacheView(k, v), mask, scale, mode=1)
    assert norm_rel(got, ref64(q16(q) if n_kv % 2 == 0 else q, k, v, mask, scale)) <= 1e-5


@pytest.mark.parametrize("T,H,Hkv,D,n_kv,prompt_kernel", [(2, 32, 8, 128, 1024, True), (2, 8, 2, 128, 1024, False), (8, 32, 32, 128, 4096, False), (12, 32, 32, 128, 4096, True),
                                                          (12, 32, 8, 128, 510, False), (16, 8, 2, 128, 512, False), (16, 32, 8, 64, 2048, True), (16, 32, 8, 64, 512, False),
                                                          (31, 32, 8, 128, 8194, False), (32, 32, 8, 128, 8194, True), (32, 8, 2, 128, 8194, False)], ids=str)
def test_which_few_rows_it_takes(dev, T, H, Hkv, D, n_kv, prompt_kernel):
    """told apart by their distance from float64: f16 weights under maxima of 16 positions (the decode kernel), or two parts"""
    q, k, v, mask = synth_case(H, Hkv, D, T, n_kv, seed=T + n_kv)
    got = dev.flash_attn(q, dev.KvCacheView(k, v), mask, D ** -0.5, mode=1)
    e = norm_rel(got, ref64(q16(q), k, v, mask, D ** -0.5))
    assert e <= 1e-5 if prompt_kernel else 2e-5 < e <= 2.5e-4
