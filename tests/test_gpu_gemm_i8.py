"""Prompt-shaped mat-muls of Q6_K, Q4_0, MXFP4 and Q8_0 weights on the tcgen05 int8 kernels (-m gpu).

Q6_K (tiled route), Q4_0 and MXFP4 (8x8 gemm route) must give the CPU oracle's bits: the kernels compute the same
exact integer block dots and run the same f32 chain.  Q8_0's tensor-core form belongs to the library's fast
numerics mode: it adds whole 32-element block dots where the CPU route adds eight lanes of four, so it is held to
the mat-mul tolerance instead, defined as the reference defines it (crates/ggml/src/compute.rs:7467-7577):
|got - ref| <= 1e-5 * sum_k |w_k x_k| per output element."""
import ctypes as C
import os
import subprocess
import sys

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
    assert dev.lib.b200_block32_kernel_choice(ty, C.c_int64(n), C.c_int64(m), 148) == columns
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


@pytest.mark.parametrize("ty", [orc.Q4_0, orc.MXFP4], ids=lambda t: orc.TYPE_NAMES[t])
def test_many_rows_of_every_code_and_far_scales(dev, ty):
    """random codes (both zeros of E2M1 among them, rows of nothing else), scales from subnormal to near the largest, activations at the ends
    of their range: the CPU route's bits"""
    n, k, m, period = 14344, 256, 509, 504
    assert dev.lib.b200_block32_kernel_choice(ty, C.c_int64(n), C.c_int64(m), 148) == 128
    rng = np.random.default_rng(460 + ty)
    if ty == orc.Q4_0:
        b = rng.integers(0, 256, (period, k // 32, 18), dtype=np.uint8)
        b[..., :2] = rng.choice(np.array([6e-8, -1e-5, 0.0, -0.0, 0.01, -0.02, 60000.0, -65504.0], np.float16), (period, k // 32)).view(np.uint8).reshape(period, k // 32, 2)
        b[5, :, 2:], b[6, :, 2:] = 0x88, 0x00
    else:
        b = rng.integers(0, 256, (period, k // 32, 17), dtype=np.uint8)
        b[..., 0] = rng.choice(np.array([0, 1, 2, 20, 118, 121, 127, 200], np.uint8), (period, k // 32))
        b[5, :, 1:], b[6, :, 1:], b[7, :, 1:] = 0x88, 0x80, 0x08
    W = b.reshape(period, -1)
    x = synth.activations(m, k, seed=461)
    x[0], x[1] = 3.0, -3.0                       # every quant 127, -127
    x[2, ::2], x[2, 1::2] = 1e-30, -1e-30
    x[3] *= 1e4
    want, _ = orc.mul_mat(ty, W, x)
    assert np.isfinite(want).all()
    W = np.tile(W, ((n + period - 1) // period, 1))[:n]
    got = dev.mul_mat(dev.Weight(ty, W, k), x)
    assert dev.kernel_error() == 0
    assert bits_equal(got, np.tile(want, (1, (n + period - 1) // period))[:, :n])


def own_block(dev, m, k):
    """a caller's activation block, 256-byte aligned"""
    buf = dev.DeviceBuffer(dev.lib.b200_act_scratch_nbytes(m, k) + 256)
    return buf, (buf.ptr + 255) // 256 * 256


@pytest.mark.parametrize("ty", [orc.MXFP4, orc.Q8_0], ids=lambda t: orc.TYPE_NAMES[t])
def test_callers_with_blocks_of_their_own_share_nothing(dev, ty):
    """two streams, each with its activation block, mat-muls side by side; a captured call replayed after larger ones"""
    import torch
    n, k, m, rounds = 14344, 1024, 509, 12
    assert dev.lib.b200_block32_kernel_choice(ty, C.c_int64(n), C.c_int64(m), 148) == 128
    w = dev.Weight(ty, synth.weights(ty, n, k, seed=440, period=504), k)
    dev.set_numerics(dev.FAST)
    try:
        jobs = []
        for i in range(2):
            x = synth.activations(m, k, seed=441 + i)
            buf, act = own_block(dev, m, k)
            jobs.append((dev.device_array(x), buf, act, dev.DeviceBuffer(4 * m * n), torch.cuda.Stream()))

        def call(job, stream):
            dx, _, act, out, _ = job
            dev.check(dev.lib.b200_quantize_activations_device(dev.ACT_Q8_0, m, k, dx.ptr, k, act, stream), "quantize")
            dev.check(dev.lib.b200_mul_mat_q8(ty, n, k, m, w.ptr, act, dev.ACT_Q8_0, out.ptr, n, 0, stream), "mul_mat_q8")

        want = []
        for job in jobs:
            call(job, None)
            want.append(job[3].download(np.uint32, m * n))
        torch.cuda.synchronize()
        before = int(dev.lib.b200_debug_alloc_count())
        for _ in range(rounds):
            for job in jobs:
                call(job, job[4].cuda_stream)
        torch.cuda.synchronize()
        assert int(dev.lib.b200_debug_alloc_count()) == before
        for job, bits in zip(jobs, want):
            assert np.array_equal(job[3].download(np.uint32, m * n), bits)

        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=jobs[0][4]):
            call(jobs[0], jobs[0][4].cuda_stream)
        big = dev.device_array(synth.activations(4 * m, k, seed=443))
        out = dev.DeviceBuffer(4 * 4 * m * n)
        dev.check(dev.lib.b200_mul_mat(ty, n, k, 4 * m, w.ptr, big.ptr, k, out.ptr, n, 0, None), "mul_mat")
        torch.cuda.synchronize()
        dev.check(dev.lib.b200_memset(jobs[0][3].ptr, 0, 4 * m * n, None), "memset")
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(jobs[0][3].download(np.uint32, m * n), want[0])
        assert dev.kernel_error() == 0
    finally:
        dev.set_numerics(dev.EXACT)


OWNED_CHILD = r"""
import b200, orc, synth
dev = b200.load()
dev.set_device(0)
dev.set_numerics(dev.FAST)
n, k, m = 14344, 1024, 509
for ty in (orc.Q8_0, orc.Q4_0, orc.MXFP4):
    w, x = dev.Weight(ty, synth.weights(ty, n, k, seed=440, period=504), k), dev.device_array(synth.activations(m, k, seed=441))
    buf, out = dev.DeviceBuffer(dev.lib.b200_act_scratch_nbytes(m, k) + 256), dev.DeviceBuffer(4 * m * n)
    act = (buf.ptr + 255) // 256 * 256
    dev.check(dev.lib.b200_quantize_activations_device(dev.ACT_Q8_0, m, k, x.ptr, k, act, None), "quantize")
    dev.check(dev.lib.b200_mul_mat_q8(ty, n, k, m, w.ptr, act, dev.ACT_Q8_0, out.ptr, n, 0, None), "mul_mat_q8")
    dev.synchronize()
print("ALLOCATED", int(dev.lib.b200_debug_alloc_count()), dev.kernel_error())
"""


def test_callers_blocks_are_all_the_memory_there_is(dev):
    """in a process whose first mat-muls these are, the library allocates nothing of its own"""
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", OWNED_CHILD], capture_output=True, text=True, cwd=here, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-3:] == ["ALLOCATED", "0", "0"], r.stdout


@pytest.mark.parametrize("kind_rows", [33, 64, 130])
@pytest.mark.parametrize("ldx_extra", [0, 3])
def test_quantized_rows_and_their_f16_form(dev, kind_rows, ldx_extra):
    """what the f16 kernel reads: the quantizer's values (held to the oracle's elsewhere) as f16 in the order 0 2 1 3 4 6 5 7 of each 8, scales by block, zero past the last row"""
    m, k = kind_rows, 768
    x = synth.activations(m, k + ldx_extra, seed=450 + m)
    x[1] = 0.0
    x[2, :64] *= 1e30
    x[3, 7] = np.nan
    x[4, 5] = np.inf
    buf, act = own_block(dev, m, k)
    dx = dev.device_array(x)
    dev.check(dev.lib.b200_quantize_activations_device(dev.ACT_Q8_0, m, k, dx.ptr, k + ldx_extra, act, None), "quantize")
    raw = buf.download(np.uint8, buf.nbytes)[act - buf.ptr:]
    blocks = np.frombuffer(dev.quantize_activations(dev.ACT_Q8_0, np.ascontiguousarray(x[:, :k])).tobytes(), np.uint8).reshape(m, k // 32, 34)
    quants = blocks[..., 2:].copy().view(np.int8).reshape(m, k)
    scales = blocks[..., :2].copy().view(np.float16).reshape(m, k // 32).astype(np.float32)
    assert np.array_equal(raw[:m * k].view(np.int8).reshape(m, k), quants)
    up = lambda v: (v + 255) // 256 * 256
    at = up(m * k) + up(m * (k // 256) * 4) + up(m * (k // 16) * 2) + up(m * (k // 32) * 2)
    order = np.array([0, 2, 1, 3, 4, 6, 5, 7])
    assert np.array_equal(raw[at:at + 2 * m * k].view(np.float16).reshape(m, k // 8, 8), quants.reshape(m, k // 8, 8)[..., order].astype(np.float16))
    at += up(2 * m * k)
    ld = (m + 127) // 128 * 128
    got = raw[at:at + 4 * ld * (k // 32)].view(np.float32).reshape(k // 32, ld)
    assert np.array_equal(got[:, :m].view(np.uint32), np.ascontiguousarray(scales.T).view(np.uint32)) and not got[:, m:].any()


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
