"""The few-rows mat-mul of the fast numerics mode (csrc/gemm_few.cu) where it can go wrong: remainders of row tiles, column blocks and groups, one and two
CTAs to a tile, walks over several tiles and matrices, the fused add, experts with no, few and many pairs (-m gpu).

Tolerance.  The operands are the oracle's quantized ones, so what differs is f32 rounding: the CPU chains take up to eight rounded operations per
256 elements, the kernel up to eight and 24 additions, each off by 2^-24 of a partial sum of at most sum |w x|: (16 K / 256 + 24) 2^-24 sum |w x|,
x as quantized (its rounding to 127 steps is common to both)."""
import ctypes as C

import numpy as np
import pytest

import b200
import orc
import synth
from conftest import bits_equal
from test_gpu_mul_mat_id import top_k_ids

pytestmark = pytest.mark.gpu
TYPES = [orc.Q4_K, orc.Q6_K, orc.Q8_0, orc.Q4_0, orc.MXFP4]


@pytest.fixture(scope="module")
def dev():
    mod = b200.load()
    assert mod.device_count() > 0
    mod.set_device(0)
    return mod


@pytest.fixture
def fast(dev):
    dev.set_numerics(dev.FAST)
    yield
    dev.set_numerics(dev.EXACT)


def bound(ty, W, k, x):
    """x: [m, k] -> [m, n]; a quantized activation is at most half a step (1/254 of its block's largest) away from its value"""
    xs = np.abs(x).reshape(-1, 32)
    xs = (xs + xs.max(axis=1, keepdims=True) / 200.0).reshape(x.shape).astype(np.float64)
    w = np.abs(orc.dequantize(ty, W, k)).astype(np.float64)
    if ty == orc.Q4_K:   # a weight is a difference of two products that the kernels sum apart
        w = w + np.abs(w).reshape(w.shape[0], -1, 256).max(axis=2).repeat(256, axis=1)
    return (16 * k / 256 + 24) * 2.0 ** -24 * (xs @ w.T) + 1e-30


def rows_for(ty, n):
    return n if ty not in (orc.Q4_0, orc.MXFP4) else (n + 7) // 8 * 8   # their few-rows kernels take the 8x8 route


@pytest.mark.parametrize("ty", TYPES, ids=lambda t: orc.TYPE_NAMES[t])
@pytest.mark.parametrize("n,k,m", [(1, 256, 2), (33, 512, 8), (32, 2048, 9), (100, 2304, 16), (64, 4352, 17), (40, 4096, 31), (6400, 512, 3), (9700, 256, 16)])
def test_edges(dev, fast, ty, n, k, m):
    """fewer groups than warps, one and two classes a warp, remainders of both; tiles with a pair of CTAs and walks of several tiles"""
    n = rows_for(ty, n)
    W = synth.weights(ty, n, k, seed=n + k, period=64)
    x = synth.activations(m, k, seed=m)
    want, _ = orc.mul_mat(ty, W, x)
    got = dev.mul_mat(dev.Weight(ty, W, k), x)
    assert dev.kernel_error() == 0
    assert (np.abs(got.astype(np.float64) - want) <= bound(ty, W, k, x)).all()


@pytest.mark.parametrize("ty", TYPES, ids=lambda t: orc.TYPE_NAMES[t])
@pytest.mark.parametrize("m", [48, 64, 100])
def test_more_rows_of_small_matrices(dev, fast, ty, m):
    """several column blocks of 16"""
    n, k = 1000, 4096
    W = synth.weights(ty, n, k, seed=5, period=64)
    x = synth.activations(m, k, seed=m)
    want, _ = orc.mul_mat(ty, W, x)
    got = dev.mul_mat(dev.Weight(ty, W, k), x)
    assert dev.kernel_error() == 0
    assert (np.abs(got.astype(np.float64) - want) <= bound(ty, W, k, x)).all()


@pytest.mark.parametrize("ty", TYPES, ids=lambda t: orc.TYPE_NAMES[t])
def test_siblings_and_the_fused_add(dev, fast, ty):
    """three matrices in one launch give the bits of three launches; result + addend is one rounded add"""
    k, m, rows = 2304, 12, (4096, 72, 1024)
    x = synth.activations(m, k, seed=6)
    Ws = [synth.weights(ty, n, k, seed=20 + i, period=64) for i, n in enumerate(rows)]
    ws = [dev.Weight(ty, W, k) for W in Ws]
    kind = dev.act_kind_for(ty, rows[0], m)
    act = dev.DeviceBuffer(dev.lib.b200_act_scratch_nbytes(m, k))
    dx = dev.device_array(x)
    dev.check(dev.lib.b200_quantize_activations_device(kind, m, k, dx.ptr, k, act.ptr, None), "quantize")
    outs = [dev.DeviceBuffer(4 * n * m) for n in rows]
    n_arr = (C.c_int64 * 3)(*rows)
    w_arr, d_arr = (C.c_void_p * 3)(*[w.ptr for w in ws]), (C.c_void_p * 3)(*[o.ptr for o in outs])
    dev.check(dev.lib.b200_mul_mat_q8_rows_multi(ty, C.c_int64(k), C.c_int64(m), 3, n_arr, w_arr, C.c_void_p(act.ptr), kind, d_arr, n_arr, None), "rows_multi")
    dev.synchronize()
    for w, o, n in zip(ws, outs, rows):
        assert bits_equal(o.download(np.float32, n * m).reshape(m, n), dev.mul_mat(w, x))
    n = rows[0]
    assert dev.lib.b200_mul_mat_q8_rows_add_fusable(ty, C.c_int64(n), C.c_int64(m)) == 1
    add = synth.activations(m, n, seed=9)
    dadd, dsum = dev.device_array(add), dev.DeviceBuffer(4 * n * m)
    dev.check(dev.lib.b200_mul_mat_q8_rows_add(ty, C.c_int64(n), C.c_int64(k), C.c_int64(m), C.c_void_p(ws[0].ptr), C.c_void_p(act.ptr), kind, C.c_void_p(outs[0].ptr), C.c_int64(n),
                                               C.c_void_p(dadd.ptr), C.c_int64(n), C.c_void_p(dsum.ptr), C.c_int64(n), None), "rows_add")
    got = outs[0].download(np.float32, n * m).reshape(m, n)
    assert bits_equal(dsum.download(np.float32, n * m).reshape(m, n), got + add)


@pytest.mark.parametrize("ty", TYPES, ids=lambda t: orc.TYPE_NAMES[t])
@pytest.mark.parametrize("experts,top,tokens,ne11,n,k", [(40, 2, 40, 1, 72, 2048), (5, 3, 30, 3, 72, 2304), (4, 4, 100, 1, 72, 1024), (60, 8, 60, 1, 400, 2048), (20, 2, 40, 1, 72, 1024)], ids=str)
def test_experts(dev, fast, ty, experts, top, tokens, ne11, n, k):
    """blocks of 8 and 16 pairs, experts without any, items that are not full; ids out of range are skipped.  (Which type takes the kernel where: MXFP4 and
    Q4_0 the first and the last two, the K-quants and Q8_0 the second and third, and the fourth.)"""
    W = synth.weights(ty, experts * n, k, seed=71, period=72 * 7 + 1).reshape(experts, n, -1)
    B = synth.activations(tokens * ne11, k, seed=72).reshape(tokens, ne11, k)
    ids = top_k_ids(tokens, experts, top, seed=73)
    if experts == 40:
        ids[ids == 7] = 8
    want, _ = orc.mul_mat_id(ty, W, B, ids)
    got = dev.mul_mat_id(dev.ExpertWeights(ty, W, n, k), B, ids)
    assert dev.kernel_error() == 0
    for t in range(tokens):
        for s in range(top):
            lim = bound(ty, W[ids[t, s]], k, B[t, s % ne11][None])[0]
            assert (np.abs(got[t, s].astype(np.float64) - want[t, s]) <= lim).all()


def exact_q6_K(W, x):
    """[m, n] in float64 over the quantized operands: six-bit codes, int8 scales, f16 and f32 factors as they are"""
    n, m, k = W.shape[0], x.shape[0], x.shape[1]
    b = W.reshape(n, -1, 210)
    lo, hi, s = b[..., :128].astype(int), b[..., 128:192].astype(int), b[..., 192:208].copy().view(np.int8).astype(np.float64)
    q = np.empty(b.shape[:2] + (2, 4, 32))
    for half in range(2):
        for part in range(4):
            byte = lo[..., 64 * half + 32 * (part & 1):][..., :32]
            q[..., half, part, :] = ((byte >> 4 if part >= 2 else byte & 15) | (hi[..., 32 * half:32 * half + 32] >> 2 * part & 3) << 4) - 32
    w = q.reshape(b.shape[:2] + (16, 16)) * s[..., None] * b[..., 208:210].copy().view(np.float16).astype(np.float64)[..., None]
    a = np.frombuffer(b"".join(np.ascontiguousarray(orc.quantize_q8_K(r)).tobytes() for r in x), np.uint8).reshape(m, -1, 292)
    a = a[..., :4].copy().view(np.float32).astype(np.float64) * a[..., 4:260].copy().view(np.int8)
    return a.reshape(m, k) @ w.reshape(n, k).T


@pytest.mark.parametrize("k", [256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("m", [8, 48])
def test_q6_k_is_no_further_from_exact_than_the_chain(dev, fast, k, m):
    """rows of a few super-blocks, where the exact kernels' chain of one fma each is the most accurate: distances over 256 x m outputs, a twentieth for
    their spread"""
    W = synth.weights(orc.Q6_K, 256, k, seed=k)
    x = synth.activations(m, k, seed=m)
    chain, route = orc.mul_mat(orc.Q6_K, W, x)
    assert route == orc.ROUTE_TILED
    want = exact_q6_K(W, x)
    got = dev.mul_mat(dev.Weight(orc.Q6_K, W, k), x)
    assert np.linalg.norm(got - want) <= 1.05 * np.linalg.norm(chain - want)


@pytest.mark.parametrize("n,k,m", [(1000, 2048, 9), (96, 1536, 16), (2048, 256, 31), (4100, 1024, 20)])
def test_q6_k_of_short_rows_keeps_the_exact_kernel(dev, fast, n, k, m):
    """9 to 31 rows of up to 8 super-blocks: the CPU's bits, as under the exact numerics"""
    W = synth.weights(orc.Q6_K, n, k, seed=n, period=64)
    x = synth.activations(m, k, seed=m)
    want, _ = orc.mul_mat(orc.Q6_K, W, x)
    assert bits_equal(dev.mul_mat(dev.Weight(orc.Q6_K, W, k), x), want)
