"""Sums whose order is part of a result.  A latent attention step against logits recorded with two pages and more per split; a selective scan of prompts
that has to give the same bits whichever of its kernels runs."""
from pathlib import Path

import numpy as np
import pytest

import zugolorn_util as zu

pytestmark = pytest.mark.gpu
RECORDED = Path(__file__).parent / "golden" / "latent_steps.npz"
CASES = {"two_splits": (192, [130, 141, 150, 163, 170, 177, 181, 188]), "three_splits": (256, [190, 193, 204, 217, 230, 252]),
         "one_sequence": (640, [577]), "sixteen": (192, list(range(129, 189, 4)) + [64])}


def latent_steps(max_context, lens):
    """Logits of four steps of a batch; every weight, token and sum comes from the seeds alone."""
    cfg = zu.config([zu.attention(heads=16, dim=40, rot_dim=16, vdim=24, kv_rank=72, window=1000)], width=64)
    w = zu.random_weights(cfg, max_context)
    seqs = [zu.tokens(n + 4, cfg["vocab"], 7 * n + b) for b, n in enumerate(lens)]
    m = zu.build(cfg, w, "bfloat16", max_batch=len(lens), max_context=max_context, max_step_tokens=4096)
    rows = [m.open() for _ in seqs]
    m.step([(r, s[:n]) for r, s, n in zip(rows, seqs, lens)], [0])
    nxt, out = np.empty(len(lens), np.int32), np.empty((4, len(lens), cfg["vocab"]), np.float32)
    for k in range(4):
        m.step_active(np.array([s[n + k] for s, n in zip(seqs, lens)], np.int32), nxt, out[k])
    m.close()
    return out


@pytest.mark.parametrize("name", CASES)
def test_latent_steps_round_as_recorded(name):
    """A split rounds its softmax weights to bf16 under its own maximum: a split per page moves these logits by 1.2e-3 to 1.7e-3 (a single sequence has many
    pages either way: not at all).  Sums in another order only turn a rounding here and there, 2^-8 of one of thousands of numbers: under 1e-4."""
    got, want = latent_steps(*CASES[name]).astype(np.float64), np.load(RECORDED)[name].astype(np.float64)
    assert np.sqrt(((got - want) ** 2).mean() / (want ** 2).mean()) < 2e-4


def test_scan_does_not_depend_on_the_batch():
    """27 blocks of 16 channels: with 12 segments more than twice the 148 SMs (two threads per channel), with 7 fewer (eight threads).  The first six
    segments lie at the same places of equally many tokens, so that only the scan differs."""
    cfg = zu.config([zu.mamba(inner=424, state=16, conv=4)], width=48)
    w = zu.random_weights(cfg, 5)
    lens = [130, 97, 64, 33, 150, 126]
    seqs = [zu.tokens(n, cfg["vocab"], n) for n in lens]
    rest = zu.tokens(120, cfg["vocab"], 1)
    got = []
    for parts in ([20] * 6, [120]):
        m = zu.build(cfg, w, "bfloat16", max_batch=12, max_step_tokens=1024)
        ends = np.concatenate([[0], np.cumsum(parts)])
        entries = seqs + [rest[a:b] for a, b in zip(ends[:-1], ends[1:])]
        _, lg = m.step([(m.open(), s) for s in entries], range(sum(lens)))
        got.append(lg.copy())
        m.close()
    assert np.array_equal(got[0], got[1])
