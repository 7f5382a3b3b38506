"""Attention of prompts in f32: a NaN among the visible keys of a row reaches its output, wherever the key lies and without a sink's weight to stand
in for it, and the rows that do not see it keep every bit."""
import numpy as np
import pytest

import vagonex_util as vu

pytestmark = pytest.mark.gpu

BAD = 5  # a token whose embedding is NaN


def logits(size, sink, toks):
    cfg = vu.config([vu.attention(heads=16, kv_heads=4, dim=24, vdim=20, rot_dims=8, size=size)], alpha=0.6)
    w = vu.random_weights(cfg, 61)
    w["l0.mix.sink"] = vu.bf16_bits(np.full(16, sink))
    w["embed"] = w["embed"].copy()
    w["embed"][BAD] = 0x7FC0
    m = vu.build(cfg, w)
    out = np.delete(vu.run_portions(m, toks, [len(toks)]), BAD, axis=1)  # (the embedding is the head too)
    m.close()
    return out


def prompt(n_bad, tokens=100):
    toks = np.array(vu.tokens(tokens, 72, 62))
    toks[toks == BAD] = BAD + 1
    toks[:n_bad] = BAD
    return toks


@pytest.mark.parametrize("sink", [-np.inf, 1.0])
@pytest.mark.parametrize("n_bad", [1, 31, 32, 33, 64])
def test_every_later_row_sees_the_nan(n_bad, sink):
    assert np.isnan(logits(None, sink, prompt(n_bad))).all()


@pytest.mark.parametrize("sink", [-np.inf, 1.0])
@pytest.mark.parametrize("size,n_bad", [(33, 32), (40, 7), (32, 32)])
def test_rows_of_later_chunks_do_not(size, n_bad, sink):
    got, clean = logits(size, sink, prompt(n_bad)), logits(size, sink, prompt(0))
    assert np.isnan(got[:size]).all()
    assert np.isfinite(clean).all() and np.array_equal(got[size:], clean[size:])
