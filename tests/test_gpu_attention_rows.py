"""Attention of prompts in f32 with enough (token, head) rows for the kernel that shares keys between eight of them: edges of its
tiles of 32 keys and of its eight rows, every mask, against the plain float64 implementation."""
import pytest

import vagonex_oracle as vo
import vagonex_util as vu
from gpu_util import assert_close

pytestmark = pytest.mark.gpu

CASES = [dict(heads=16, kv_heads=16, dim=4, vdim=5, rot_dims=2, size=None), dict(heads=24, kv_heads=8, dim=33, vdim=31, rot_dims=6, size=32),
         dict(heads=20, kv_heads=4, dim=64, vdim=128, rot_dims=64, size=33), dict(heads=18, kv_heads=2, dim=128, vdim=129, rot_dims=0, size=None),
         dict(heads=16, kv_heads=1, dim=130, vdim=256, rot_dims=20, size=70)]


@pytest.mark.parametrize("kw", CASES, ids=lambda k: "-".join(map(str, k.values())))
@pytest.mark.parametrize("sizes", [[100], [75, 76], [31, 97]], ids=str)
def test_rows_that_share_keys(kw, sizes):
    cfg = vu.config([vu.attention(**kw)], alpha=0.6)
    w, toks = vu.random_weights(cfg, 51), vu.tokens(sum(sizes), 72, 52)
    m = vu.build(cfg, w)
    assert_close(vu.run_portions(m, toks, sizes), vo.forward(cfg, vu.oracle_weights(w), toks), 4e-5)  # (the bar of the other fp32 models)
    m.close()


@pytest.mark.parametrize("size", [None, 33, 40, 70])
@pytest.mark.parametrize("heads,kv_heads", [(16, 16), (16, 4), (16, 1)])
def test_a_sink_that_is_switched_off(heads, kv_heads, size):
    """A sink of -inf has no weight, also in a row whose keys all lie in the second group's tiles (a later chunk than that of the rows beside it)."""
    import numpy as np
    cfg = vu.config([vu.attention(heads=heads, kv_heads=kv_heads, dim=24, vdim=20, rot_dims=8, size=size)], alpha=0.6)
    w, toks = vu.random_weights(cfg, 53), vu.tokens(100, 72, 54)
    w["l0.mix.sink"] = vu.bf16_bits(np.where(np.arange(heads) % 3 == 2, 0.5, -np.inf))
    m = vu.build(cfg, w)
    assert_close(vu.run_portions(m, toks, [100]), vo.forward(cfg, vu.oracle_weights(w), toks), 4e-5)  # (the bar of the other fp32 models)
    m.close()
