"""Sums whose order is part of a result.  A latent attention step against logits recorded with two pages and more per split; a selective scan of prompts
that has to give the same bits whichever of its kernels runs; the sum of squares of the final norm."""
from pathlib import Path

import numpy as np
import pytest

import vagonex_util as vu
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


@pytest.mark.parametrize("width", [40, 520, 1032, 4096, 4104])
def test_sum_of_squares_of_the_final_norm(width):
    """Component c belongs to thread c % 256, a warp's sums meet in exchanges from 16 down, the warps' sums in order: with an embedding whose first rows are
    those of the identity the logits are the normed row, bit for bit."""
    import torch
    rng = np.random.default_rng(width)
    n = 40
    embed = np.concatenate([np.eye(width), rng.standard_normal((n, width))]).astype(np.float32)
    cfg = vu.config([vu.lightning(heads=1, dim=8, vdim=8)], width=width, vocab=width + n, alpha=1.0, scale=1.0, eps=1e-6)
    gain = rng.standard_normal(width).astype(np.float32)
    w = {"embed": embed, "final.norm": gain, "l0.norm1": np.ones(width, np.float32), "l0.mix.norm": np.ones(8, np.float32)}
    w.update({"l0.mix." + s: np.zeros((8, width), np.float32) for s in "qkvg"}, **{"l0.mix.o": np.zeros((width, 8), np.float32)})
    m = vu.build(cfg, w, "float32", max_batch=1, max_context=64, max_step_tokens=64)
    tap = torch.zeros(1, n, width, device="cuda")
    m.set_tap(tap)
    _, lg = m.step([(m.open(), list(range(width, width + n)))], range(n))
    m.close()
    x = tap[0].cpu().numpy()
    f32 = np.float32
    part = np.zeros((n, 256), f32)
    for c0 in range(0, width, 256):
        v = x[:, c0:c0 + 256].astype(np.float64)
        part[:, :v.shape[1]] = (v * v + part[:, :v.shape[1]]).astype(f32)
    lanes = part.reshape(n, 8, 32)
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[..., np.arange(32) ^ o]
    total = np.zeros(n, f32)
    for k in range(8):
        total = total + lanes[:, k, 0]
    rms = np.sqrt(total / f32(width) + f32(1e-6))
    assert np.array_equal(lg[:, :width], x / rms[:, None] * gain)
