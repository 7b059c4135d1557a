"""What a decode call moves and reports: logits in pieces through page-locked slots, a step's inputs by one kernel from page-locked memory or, where that
does not take them, by copies, and an error code that a kernel left (-m gpu)."""
import ctypes as C
import importlib
import os
import subprocess
import sys

import numpy as np
import pytest

import b200
import ggml_plugin as gp
from conftest import bits_equal
from test_gpu_llama import SMALL, both, make_model, run_sequence

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ll():
    b200.load()
    return importlib.import_module("llama_rust_b200.llama")


@pytest.mark.parametrize("rows", [1, 2, 9, 20])
def test_logits_of_a_large_vocabulary(ll, rows):
    """31990 values a row: part of a slot, one and a bit, all four, each of them taken more than once with a ragged last piece; against the tensor as a
    plain copy reads it"""
    hp = dict(SMALL, n_vocab=31990, n_layer=1)
    gpu, _ = both(ll, hp, make_model(ll, hp, 51), 256, 32)
    toks = np.arange(100, 100 + rows)
    for at in (0, rows):   # the slots are used again by the next call
        got, am = gpu.decode_seqs(toks + at, np.arange(at, at + rows), [0] * rows, np.arange(rows), argmax=True)
        want = gpu.read_node("result_output", 31990 * rows).reshape(rows, 31990)
        assert bits_equal(got, want)
        assert (am == want.argmax(axis=1)).all()
    gpu.close()


def test_a_mask_larger_than_the_page_locked_block(ll):
    """400 rows x 512 cells of 2 bytes: by a copy of its own beside the others' kernel; the CPU's bits"""
    run_sequence(ll, SMALL, seed=61, prompt_len=400, n_gen=2, n_ctx=1024)


@pytest.fixture
def sess():
    lib, reg = gp.load_backend(b200.load().LIB_PATH)
    s = gp.Session(lib, reg)
    yield s
    s.close()


def test_inputs_of_every_kind(sess):
    """more tensors than a launch carries, odd numbers of words, destinations off 16 bytes, bytes that are not whole words, one larger than the block, and
    all that again with other values while the first lot may still be on its way"""
    fn = sess.reg.contents.iface.get_proc_address(sess.regp, b"b200_backend_set_inputs")
    set_inputs = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_int, C.POINTER(C.POINTER(gp.Tensor)), C.POINTER(C.c_void_p), C.POINTER(C.c_size_t))(fn)
    sizes = [1, 3, 4, 5, 1023, 1024, 4099, 9000, 2, 7, 16, 31, 33, 64, 100]   # 15 tensors of F32: 12 at a time by the kernel
    tensors = [sess.new_tensor(gp.F32, [n]) for n in sizes]
    off = sess.new_tensor(gp.F32, [64])
    off.data = off.data + 4          # a view that begins between 16-byte boundaries
    off.ne[0], off.nb[1], off.nb[2], off.nb[3] = 61, 244, 244, 244
    halves = sess.new_tensor(gp.F16, [7])
    large = sess.new_tensor(gp.F32, [50000])
    order = [off, halves, large] + tensors
    rng = np.random.default_rng(5)
    for lot in range(3):
        arrs = [rng.integers(0, 1 << 32, int(t.ne[0]), dtype=np.uint64).astype(np.uint32) if t is not halves else rng.integers(0, 1 << 16, 7).astype(np.uint16) for t in order]
        ptrs = (C.POINTER(gp.Tensor) * len(order))(*[C.pointer(t) for t in order])
        data = (C.c_void_p * len(order))(*[a.ctypes.data for a in arrs])
        size = (C.c_size_t * len(order))(*[a.nbytes for a in arrs])
        assert set_inputs(sess.bep, len(order), ptrs, data, size) == 0
        wants = [a.copy() for a in arrs]
        for a in arrs:
            a[:] = 0                 # the sources are free on return
        if lot == 1:
            continue                 # nothing reads this lot: the next follows at once
        sess.be.iface.synchronize(sess.bep)
        for t, want in zip(order, wants):
            assert (sess.get(t, want.dtype, want.size) == want).all()


def test_an_error_code_that_another_thread_clears(tmp_path):
    """A step whose kernel gave up reports the code that came behind its logits, also when the device's word has been read and cleared by another context
    before the step clears it: a b200_kernel_error that finds nothing stands in for that."""
    src, so = tmp_path / "cleared.c", tmp_path / "cleared.so"
    src.write_text("int b200_kernel_error(int *code) { *code = 0; return 0; }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    child = """
import importlib, sys
import numpy as np
import b200
from test_gpu_llama import SMALL, both, make_model
dev = b200.load()
ll = importlib.import_module("llama_rust_b200.llama")
dev.set_device(0)
dev.set_numerics(dev.FAST)
hp = dict(SMALL, n_layer=1)
gpu, _ = both(ll, hp, make_model(ll, hp, 3), 256, 8)
gpu.decode_seqs([1, 2], [0, 1], [0, 0], [0, 1])
dev.lib.b200_debug_few_rows_wait(20000, 0)
try:
    gpu.decode_seqs([3, 4, 5], [2, 3, 4], [0, 0, 0], [0, 1, 2])
except dev.B200Error as e:
    assert "error code 4" in str(e), e
    print("reported")
finally:
    dev.lib.b200_debug_few_rows_wait(0, -1)
"""
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", child], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "reported" in r.stdout
