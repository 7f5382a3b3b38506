"""Attention of prompts with enough (token, head) rows for the kernel that shares keys between sixteen of them: edges of its tiles of 32 keys and of its
sixteen rows (two per warp), every mask, one and two groups of warps, against the plain float64 implementation."""
import numpy as np
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
    cfg = vu.config([vu.attention(heads=heads, kv_heads=kv_heads, dim=24, vdim=20, rot_dims=8, size=size)], alpha=0.6)
    w, toks = vu.random_weights(cfg, 53), vu.tokens(100, 72, 54)
    w["l0.mix.sink"] = vu.bf16_bits(np.where(np.arange(heads) % 3 == 2, 0.5, -np.inf))
    m = vu.build(cfg, w)
    assert_close(vu.run_portions(m, toks, [100]), vo.forward(cfg, vu.oracle_weights(w), toks), 4e-5)  # (the bar of the other fp32 models)
    m.close()


@pytest.mark.parametrize("dtype,tol", [("float32", 4e-5), ("bfloat16", 0.08)])  # (the bars of the other models of these types)
@pytest.mark.parametrize("dim,vdim", [(256, 256), (320, 128), (300, 120), (320, 250)])
@pytest.mark.parametrize("sizes,size", [([75, 76], None), ([100], 33)], ids=str)
def test_heads_too_wide_for_two_groups(dim, vdim, sizes, size, dtype, tol):
    """Two tiles of keys and values for each of two groups of warps would not fit in shared memory: one group (bf16 heads up to 256 wide run on the tensor cores)."""
    cfg = vu.config([vu.attention(heads=16, kv_heads=4, dim=dim, vdim=vdim, rot_dims=32, size=size)], alpha=0.6)
    w, toks = vu.random_weights(cfg, 55), vu.tokens(sum(sizes), 72, 56)
    m = vu.build(cfg, w, dtype)
    got, want = vu.run_portions(m, toks, sizes), vo.forward(cfg, vu.oracle_weights(w), toks)
    assert vu.error(got, want) < tol
    m.close()
