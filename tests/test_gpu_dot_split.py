"""fp32 products on the tensor cores (dot_split.cu) against float64: the vocabulary projection of an f32 model whose layers pass the token through, so that the
operands are known: on both sides of the lines of its dispatch (33 tokens, a million weights), at both edges of the token tiles of 32 / 64 / 96 / 128, of the feature tile of 128 and of the blocks of 64 products,
with clusters of one to eight CTAs; weights of 24 bits and weights that fit bf16; infinities, NaN and numbers beyond bf16's range."""
import numpy as np
import pytest

import vagonex_oracle as vo
import vagonex_util as vu
import zugolorn_oracle as zo
import zugolorn_util as zu

pytestmark = pytest.mark.gpu


def head_model(width, embed, T):
    """A model whose sublayers add nothing: the operand of the vocabulary projection is the normed embedding."""
    vocab = embed.shape[0]
    cfg = vu.config([vu.lightning(heads=1, dim=8, vdim=8)], width=width, vocab=vocab, alpha=1.0, scale=1.0, eps=1e-6)
    w = {"embed": embed, "final.norm": np.ones(width, np.float32), "l0.norm1": np.ones(width, np.float32), "l0.mix.norm": np.ones(8, np.float32)}
    for s in "qkvg":
        w["l0.mix." + s] = np.zeros((8, width), np.float32)
    w["l0.mix.o"] = np.zeros((width, 8), np.float32)
    return vu.build(cfg, w, "float32", max_batch=1, max_context=512, max_step_tokens=512)


def operand(embed, toks):
    x = embed[toks].astype(np.float64)
    for _ in range(2):
        x = x / np.sqrt((x * x).mean(-1, keepdims=True) + 1e-6)
    return x


def logits(m, toks):
    row = m.open()
    _, lg = m.step([(row, toks)], range(len(toks)))
    m.retire(row)
    return lg


def check(got, x, w):
    """Every addition of a block truncates (24 per block at most), the others round: 2^-19 of the sum of magnitudes covers them and the two norms."""
    want, size = x @ w.T, np.abs(x) @ np.abs(w).T
    assert np.all(np.abs(got - want) <= 2.0 ** -19 * size)
    # and on the whole no further off than fp32 additions in any order
    assert np.sqrt(((got - want) ** 2).mean() / (want ** 2).mean()) < 5e-7


@pytest.mark.parametrize("kind", ["full", "bf16", "mixed"])
@pytest.mark.parametrize("T,vocab,width", [(1, 1024, 1024), (17, 7712, 136), (32, 4097, 264), (32, 1016, 1032), (33, 40, 8), (64, 128, 64), (65, 136, 72), (96, 300, 1032), (97, 1000, 136), (128, 260, 520), (129, 2049, 200), (250, 1003, 2056)])
def test_against_float64(T, vocab, width, kind):
    rng = np.random.default_rng(T * vocab)
    embed = rng.standard_normal((vocab, width)).astype(np.float32)
    short = (embed.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)
    if kind == "bf16":
        embed = short
    elif kind == "mixed":  # blocks with and without further parts, next to each other
        pick = rng.random((vocab // 32 + 1, width // 64 + 1)) < 0.5
        embed = np.where(np.repeat(np.repeat(pick, 32, 0), 64, 1)[:vocab, :width], embed, short)
    toks = rng.integers(0, vocab, T)
    m = head_model(width, embed, T)
    check(logits(m, toks), operand(embed, toks), embed.astype(np.float64))
    m.close()


def test_numbers_that_do_not_split():
    rng = np.random.default_rng(3)
    embed = rng.standard_normal((200, 136)).astype(np.float32)
    toks = rng.integers(0, 150, 70)  # (the rows behind are only features)
    embed[150, 7], embed[151, 9], embed[152, 100] = np.inf, np.nan, -np.inf
    embed[153, [1, 2]] = np.inf, -np.inf
    embed[154:160] = 0.0
    embed[154, 135], embed[155, 0], embed[156, 64] = 3.4e38, -3.39e38, 1e-38
    m = head_model(136, embed, 70)
    got, x = logits(m, toks), operand(embed, toks)
    with np.errstate(all="ignore"):
        want = (x @ embed.astype(np.float64).T).astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fine = np.isfinite(want)
    assert fine[:, 154].any() and np.isinf(want[:, 154]).any()
    assert np.allclose(got[fine], want[fine], rtol=2e-5, atol=2e-5)
    assert np.allclose(got[:, 156], want[:, 156], rtol=1e-5, atol=2.0 ** -133)
    m.close()


@pytest.mark.parametrize("T,width,ff", [(33, 40, 20), (64, 64, 64), (70, 72, 72), (129, 136, 200), (40, 200, 1000), (5, 520, 1016), (300, 64, 129)])
@pytest.mark.parametrize("design", ["vagonex", "zugolorn"])
def test_gate_up_pairs(design, T, width, ff):
    """A feed-forward in one launch of pairs: tiles of 64 features and their remainders, both activations, weights of 24 bits, against the whole model in float64."""
    if design == "vagonex":
        util, forward = vu, vo.forward
        cfg = vu.config([vu.lightning(heads=2, dim=12, vdim=12, ff=ff)], width=width)
    else:
        util, forward = zu, zo.forward
        cfg = zu.config([zu.mamba(inner=48, ff=ff, limit=0.8)], width=width)
    rng = np.random.default_rng(ff)
    w = {k: vu.widen(v).astype(np.float32) for k, v in util.random_weights(cfg, T).items()}
    for k in w:  # (numbers that bf16 does not hold; the zeros of a design stay)
        w[k] = np.where(w[k] == 0, w[k], w[k] * (1 + 2.0 ** -9 * rng.standard_normal(w[k].shape))).astype(np.float32)
    toks = vu.tokens(T, cfg["vocab"], T)
    m = util.build(cfg, w, "float32")
    got = logits(m, toks)
    assert util.error(got, forward(cfg, {k: v.astype(np.float64) for k, v in w.items()}, toks)) < 4e-5  # (the bar of the other fp32 models)
    m.close()


def products(x, w, scale_x=1.0, scale_w=1.0):
    """x . w^T scaled by powers of two, as a model's logits, and what float64 makes of the very operands: a second model, whose vocabulary has the rows of
    the identity, shows the normed x bit for bit."""
    (T, K), eye = x.shape, np.eye(x.shape[1], dtype=np.float32)
    out = []
    for embed, gain, toks in ((np.concatenate([eye, x]), 1.0, K + np.arange(T)), (np.concatenate([x, w * np.float32(scale_w)]), scale_x, np.arange(T))):
        cfg = vu.config([vu.lightning(heads=1, dim=8, vdim=8)], width=K, vocab=len(embed), alpha=1.0, scale=1.0, eps=1e-6)
        ws = {"embed": embed, "final.norm": np.full(K, gain, np.float32), "l0.norm1": np.ones(K, np.float32), "l0.mix.norm": np.ones(8, np.float32), "l0.mix.o": np.zeros((K, 8), np.float32)}
        ws.update({"l0.mix." + n: np.zeros((8, K), np.float32) for n in "qkvg"})
        m = vu.build(cfg, ws, "float32", max_batch=1, max_context=512, max_step_tokens=512)
        out.append(logits(m, toks).astype(np.float64))
        m.close()
    normed = out[0][:, :K] * scale_x
    return out[1][:, T:], normed @ (w.astype(np.float64) * scale_w).T


def rms(got, want):
    return float(np.sqrt(((got - want) ** 2).mean() / (want ** 2).mean()))


@pytest.mark.parametrize("T,K", [(40, 64), (40, 200), (128, 520), (40, 1024), (128, 2752)])
@pytest.mark.parametrize("kind", ["positive", "bf16 weights", "mantissas"])
def test_operands_of_one_sign(kind, T, K):
    """Nothing cancels: the truncated additions of the tensor core all err to the same side, a quarter to a half of 2^-24 each time an accumulator is
    finished, and the left-out products m l and l m are 2^-24 of the product together at worst (mantissas just below a bf16 midpoint).  With a rounding
    or two of 2^-25 on the whole sum that is under 2^-24; the additions of fp32 chains stay between 4.5e-8 and 8e-8 here."""
    rng = np.random.default_rng(T * K)
    x, w = np.abs(rng.standard_normal((T, K))).astype(np.float32), np.abs(rng.standard_normal((256, K))).astype(np.float32)
    if kind == "bf16 weights":
        w = (w.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)
    elif kind == "mantissas":
        x, w = (np.float32(1.00390625 - 2.0 ** -17) * 2.0 ** rng.integers(-1, 2, a.shape) for a in (x, w))
    assert rms(*products(x.astype(np.float32), w.astype(np.float32))) < 2.0 ** -24


@pytest.mark.parametrize("scale_x,scale_w", [(1.0, 2.0 ** -118), (2.0 ** -118, 2.0 ** 20), (2.0 ** -60, 2.0 ** -60), (2.0 ** -20, 2.0 ** 100), (1.0, 2.0 ** 110)])
@pytest.mark.parametrize("T,K", [(9, 1032), (64, 136)])
def test_operands_far_from_one(T, K, scale_x, scale_w):
    """Powers of two change nothing: no part of a small number is lost, and what leaves bf16's range is formed again in fp32.  The bar is that of operands around
    one, fp32 additions of random signs (1.1e-7 for chains of this length)."""
    rng = np.random.default_rng(K)
    x, w = rng.standard_normal((T, K)).astype(np.float32), rng.standard_normal((1024 if T < 33 else 72, K)).astype(np.float32)
    assert rms(*products(x, w, scale_x, scale_w)) < 1.1e-7


def test_a_few_small_numbers_among_others():
    """A product's rows with numbers of all magnitudes: each result against the sum of its own magnitudes."""
    rng = np.random.default_rng(8)
    x, w = rng.standard_normal((40, 136)).astype(np.float32), rng.standard_normal((96, 136)) * 2.0 ** rng.integers(-125, 3, (96, 136))
    w[:48] *= 2.0 ** -20  # subnormal ones among them
    w = w.astype(np.float32)
    got, want = products(x, w)
    size = np.abs(want).max(axis=0)  # (of a feature)
    assert np.all(np.abs(got - want).max(axis=0) <= 2.0 ** -21 * size + 2.0 ** -148)

