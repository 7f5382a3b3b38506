"""Recurrences that walk their tokens one by one (f32 models, and wide heads of bf16 ones) against float64, for segments that end around a turn of
staged tokens (16, and 8 for more than 128 key components), every width of a thread's rows, and value columns that end inside a block."""
import numpy as np
import pytest

import vagonex_oracle as vo
import vagonex_util as vu

pytestmark = pytest.mark.gpu
LENS = [1, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 70]


@pytest.mark.parametrize("dim,vdim", [(24, 8), (64, 20), (128, 36), (136, 16), (256, 9)])
@pytest.mark.parametrize("kind", ["delta", "lightning"])
def test_segments_around_a_turn(kind, dim, vdim):
    layer = vu.delta(heads=2, kv_heads=1, dim=dim, vdim=vdim) if kind == "delta" else vu.lightning(heads=2, dim=dim, vdim=vdim)
    cfg = vu.config([layer], width=64)
    w = vu.random_weights(cfg, dim + vdim)
    seqs = [vu.tokens(n + 5, cfg["vocab"], n) for n in LENS]
    want = [vo.forward(cfg, vu.oracle_weights(w), s) for s in seqs]
    for dtype, tol in (("float32", 4e-5), ("bfloat16", 0.08)):  # as for the other recurrences of these models (test_gpu_vagonex.py)
        if dtype == "bfloat16" and dim <= 128:
            continue  # these prompts go through the chunks
        m = vu.build(cfg, w, dtype, max_batch=len(LENS), max_step_tokens=512)
        rows = [m.open() for _ in seqs]
        for hi in (0, 5):  # the prompts, then five tokens more: a state that goes on
            parts = [s[:n] if hi == 0 else s[n:n + 5] for s, n in zip(seqs, LENS)]
            ends = np.cumsum([len(p) for p in parts])
            places = sorted({int(e) - 1 - k for e, p in zip(ends, parts) for k in (0, len(p) // 2)})
            _, lg = m.step(list(zip(rows, parts)), places)
            ref = np.concatenate([o[:n] if hi == 0 else o[n:n + 5] for o, n in zip(want, LENS)])[places]
            assert vu.error(lg, ref) < tol, (dtype, hi)
        m.close()
