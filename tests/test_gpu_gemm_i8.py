"""Prompt-shaped mat-muls of Q6_K, Q4_0, MXFP4 and Q8_0 weights on the tcgen05 int8 kernels (-m gpu).

Q6_K (tiled route), Q4_0 and MXFP4 (8x8 gemm route) must give the CPU oracle's bits: the kernels compute the same
exact integer block dots and run the same f32 chain.  Q8_0's tensor-core form belongs to the library's fast
numerics mode: it adds whole 32-element block dots where the CPU route adds eight lanes of four, so it is held to
the mat-mul tolerance instead, defined as the reference defines it (crates/ggml/src/compute.rs:7467-7577):
|got - ref| <= 1e-5 * sum_k |w_k x_k| per output element."""
import ctypes as C

import numpy as np
import pytest

import b200
import orc
import synth
from conftest import bits_equal

pytestmark = pytest.mark.gpu

SHAPES = [(256, 1024, 40), (128, 256, 32), (300, 2048, 33), (1024, 4096, 100), (4096, 4096, 512), (96, 512, 8)]


@pytest.fixture(scope="module")
def dev():
    mod = b200.load()
    assert mod.device_count() > 0
    mod.set_device(0)
    return mod


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("ty", [orc.Q6_K, orc.Q4_0, orc.MXFP4], ids=lambda t: orc.TYPE_NAMES[t])
def test_bit_exact_types(dev, ty, shape, monkeypatch):
    n, k, m = shape
    if ty != orc.Q6_K and n % 8:
        pytest.skip("the 8x8 route needs rows % 8 == 0")
    W = synth.weights(ty, n, k, seed=400 + ty, period=512)
    x = synth.activations(m, k, seed=401 + m)
    want, _ = orc.mul_mat(ty, W, x)
    # Q6_K takes its tcgen05 kernel only on request (the mma.sync kernel is the quicker one): ask for it here
    monkeypatch.setenv("B200_Q6K_TCGEN05", "1")
    got = dev.mul_mat(dev.Weight(ty, W, k), x)
    assert dev.kernel_error() == 0
    assert bits_equal(got, want), f"max |d| = {np.abs(got - want).max()}"


# the f16 kernel's tiles of 64 and of 128 columns, ragged on both sides: one tile a CTA, then three and more (its stages, scale slots and sums
# carried from tile to tile), the last ones with only one 256-element group a tile
MANY_ROWS = [(2056, 4096, 300, 64), (2000, 2048, 705, 128), (4728, 2816, 193, 64), (56296, 1024, 61, 64), (14344, 1024, 509, 128), (14344, 256, 509, 128)]


@pytest.mark.parametrize("shape", MANY_ROWS, ids=lambda s: "x".join(map(str, s[:3])))
@pytest.mark.parametrize("ty", [orc.Q4_0, orc.MXFP4, orc.Q8_0], ids=lambda t: orc.TYPE_NAMES[t])
def test_many_rows(dev, ty, shape):
    n, k, m, columns = shape
    assert dev.lib.b200_block32_kernel_choice(ty, C.c_int64(n), C.c_int64(k), C.c_int64(m), 148) == columns
    period, ld = 504, n + 8   # rows of the result farther apart than its length
    W = synth.weights(ty, n, k, seed=420 + ty, period=period)
    x = synth.activations(m, k, seed=421 + m)
    want, _ = orc.mul_mat(ty, W[:period], x)   # a multiple of 8 rows: the same route
    want = np.tile(want, (1, (n + period - 1) // period))[:, :n]
    w, dx, out = dev.Weight(ty, W, k), dev.device_array(x), dev.device_array(np.full((m, ld), 7.0, np.float32))

    def run(entry):
        dev.check(entry(ty, n, k, m, w.ptr, dx.ptr, k, out.ptr, ld, 0, None), "mul_mat")
        assert dev.kernel_error() == 0
        got = out.download(np.float32, m * ld).reshape(m, ld)
        assert (got[:, n:] == 7.0).all()
        return got[:, :n]

    dev.set_numerics(dev.FAST)
    try:
        got = run(dev.lib.b200_mul_mat)
        if ty != orc.Q8_0:
            assert bits_equal(got, want)
        elif dev.lib.b200_act_scratch_nbytes(m, k) <= dev.lib.b200_static_scratch_nbytes():
            assert bits_equal(got, run(dev.lib.b200_mul_mat_static_scratch))   # the int8 kernel: the same chain
    finally:
        dev.set_numerics(dev.EXACT)
    bound = 1e-5 * (np.abs(x).astype(np.float64) @ np.abs(orc.dequantize(ty, W[:period], k)).astype(np.float64).T)
    bound = np.tile(bound, (1, (n + period - 1) // period))[:, :n]
    assert (np.abs(got.astype(np.float64) - want.astype(np.float64)) <= bound).all()


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_q8_0_fast_mode_within_the_mat_mul_tolerance(dev, shape):
    n, k, m = shape
    W = synth.weights(orc.Q8_0, n, k, seed=410, period=512)
    x = synth.activations(m, k, seed=411 + m)
    want, _ = orc.mul_mat(orc.Q8_0, W, x)
    dev.set_numerics(dev.FAST)
    try:
        got = dev.mul_mat(dev.Weight(orc.Q8_0, W, k), x)
    finally:
        dev.set_numerics(dev.EXACT)
    assert dev.kernel_error() == 0
    bound = 1e-5 * (np.abs(x).astype(np.float64) @ np.abs(orc.dequantize(orc.Q8_0, W, k)).astype(np.float64).T)
    err = np.abs(got.astype(np.float64) - want.astype(np.float64))
    assert (err <= bound).all(), f"worst ratio to the bound: {(err / bound).max():.3g}"
    print(f"Q8_0 {shape}: max |got - ref| / sum|w x| = {(err / (bound * 1e5)).max():.2e}")
    # and in exact mode the same call reproduces the CPU's lanes
    assert bits_equal(dev.mul_mat(dev.Weight(orc.Q8_0, W, k), x), want)
