"""Grouped-query attention of long prompts on tcgen05 (csrc/grouped_attn_tcgen05.cu) against the plain restatement: head sizes 64 and 128, groups of
one to eight query heads, windows and kept positions that end inside tiles, queries rotated in pairs and not, several sequences in a step, cells
that stand in runs and cells that do not (-m gpu).  BF16 models; limits as in test_gpu_lenolix.py (decoder_checks.Expected)."""
import importlib

import numpy as np
import pytest

import b200
import lenolix_models as M
from decoder_checks import Expected, check, feed, model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ll():
    b200.load()
    return importlib.import_module("llama_rust_b200.llama")


CASES = {
    "128, four heads a key head": M.layer(heads=8, kv_heads=2, dim=128, vdim=128, window=130, keep=9, rot=64),
    "128, a head each, everything rotates": M.layer(heads=2, kv_heads=2, dim=128, vdim=128, window=64, keep=70, rot=128, scaling=None),
    "128, eight heads on one, no window": M.layer(heads=8, kv_heads=1, dim=128, vdim=128, window=None, rot=32),
    "128, rotated pairs off 16 bytes": M.layer(heads=4, kv_heads=2, dim=128, vdim=128, window=200, keep=0, rot=70, scaling=None),
    "64, two heads a key head": M.layer(heads=4, kv_heads=2, dim=64, vdim=64, window=128, keep=128, rot=64),
    "64, nothing rotates": M.layer(heads=4, kv_heads=1, dim=64, vdim=64, window=1, keep=1, rot=0, scaling=None),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("n", [256, 333])
def test_prompts(ll, name, n):
    cfg = M.config([CASES[name]], width=64)
    w, toks = M.weights(cfg, 7), M.tokens(cfg, n, 8)
    m = model(ll, cfg, w, "bfloat16")
    check(feed(m, toks, n), Expected(cfg, w, toks, "bfloat16"), name)


def test_sequences_side_by_side_and_a_continuation(ll):
    """two prompts in one step, then the second half of a longer one over cells of an earlier step"""
    cfg = M.config([CASES["128, four heads a key head"]], width=64)
    w = M.weights(cfg, 17)
    toks = [M.tokens(cfg, n, 18 + n) for n in (150, 140, 300)]
    want = [Expected(cfg, w, t, "bfloat16") for t in toks]
    m = model(ll, cfg, w, "bfloat16", n_ctx=768)
    rows, pos, seq = list(toks[0]) + list(toks[1]), list(range(150)) + list(range(140)), [0] * 150 + [1] * 140
    got, _ = m.decode_seqs(rows, pos, seq, np.arange(290))
    check(got[:150], want[0], "first")
    check(got[150:], want[1], "second")
    check(feed(m, toks[2][:40], 40, 2), want[2][:40], "beginning")
    check(feed(m, toks[2][40:], 260, 2, 40), want[2][40:], "continuation")


def test_cells_that_do_not_stand_together(ll):
    """every other cell is taken by another sequence"""
    cfg = M.config([CASES["128, eight heads on one, no window"]], width=64)
    w = M.weights(cfg, 27)
    toks = M.tokens(cfg, 280, 28)
    m = model(ll, cfg, w, "bfloat16", n_ctx=768)
    a, b = M.tokens(cfg, 100, 29), M.tokens(cfg, 100, 30)
    for i in range(100):
        m.decode_seqs([a[i], b[i]], [i, i], [0, 1], [0])
    m.seq_rm(0)
    check(feed(m, toks, 280, 2), Expected(cfg, w, toks, "bfloat16"), "holes")


@pytest.mark.parametrize("name", ["128, four heads a key head", "128, a head each, everything rotates", "64, two heads a key head"])
def test_a_token_of_nan(ll, name):
    """its query, key and value are NaN: the rows that see it are NaN (sinks or not), those before it and those that it has left the window of keep
    what they are without it, in the tiles that hold it too"""
    cfg = M.config([dict(CASES[name], mlp=None)], width=64, bigram=None)
    w = M.weights(cfg, 37)
    toks = np.array(M.tokens(cfg, 400, 38))
    toks[toks == 100] = 99
    bad = 170
    clean = Expected(cfg, w, toks, "bfloat16")
    toks[bad] = 100
    w["embed"] = w["embed"].copy()
    w["embed"][100, 3] = np.nan
    mask = CASES[name]["mixer"]["mask"]
    sees = np.array([i >= bad and i - bad < mask["size"] for i in range(400)])
    got = feed(model(ll, cfg, w, "bfloat16"), toks, 400)[:, :100]   # (token 100's own logit is NaN in every row)
    assert np.isnan(got[sees]).all() and np.isfinite(got[~sees]).all()
    e = M.error(got[~sees], clean.rows[~sees][:, :100])
    assert (e < clean.limit[~sees]).all()
