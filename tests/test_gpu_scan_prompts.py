"""Selective scans of bf16 prompts against float64 on both sides of the rule that chooses between their kernels (blocks of 16 channels per segment against
two per SM), for segments that end around a tile of 32 tokens or eight, channels that end inside a block of 64, and 9 to 16 states."""
import numpy as np
import pytest

import zugolorn_oracle as zo
import zugolorn_util as zu

pytestmark = pytest.mark.gpu
LENS = [1, 7, 8, 9, 31, 32, 33, 40, 63, 64, 65, 97]


@pytest.mark.parametrize("inner,state", [(424, 16), (424, 9), (420, 13), (400, 17), (384, 16), (392, 8)])
def test_segments_around_a_tile(inner, state):
    """12 segments: 25 blocks of 16 channels each are 300, more than twice the 148 SMs; 24 are 288."""
    cfg = zu.config([zu.mamba(inner=inner, state=state, conv=4)], width=48)
    w = zu.random_weights(cfg, inner + state)
    seqs = [zu.tokens(n + 41, cfg["vocab"], n) for n in LENS]
    want = [zo.forward(cfg, zu.oracle_weights(w), s) for s in seqs]
    m = zu.build(cfg, w, "bfloat16", max_batch=len(LENS), max_step_tokens=1024)
    rows = [m.open() for _ in seqs]
    for more in (0, 41):  # the prompts, then 41 tokens more: a state that goes on
        parts = [s[n:n + more] if more else s[:n] for s, n in zip(seqs, LENS)]
        ends = np.cumsum([len(p) for p in parts])
        places = sorted({int(e) - 1 - k for e, p in zip(ends, parts) for k in (0, len(p) // 2, len(p) - 1)})
        _, lg = m.step(list(zip(rows, parts)), places)
        ref = np.concatenate([o[n:n + more] if more else o[:n] for o, n in zip(want, LENS)])[places]
        assert zu.error(lg, ref) < 0.08, more  # bf16 models (test_gpu_zugolorn.py)
    m.close()
