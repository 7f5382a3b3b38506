"""Decode steps of the layer-list decoder against float64 at the sizes where their kernels change form: batches around 8 and 16 (the merge of the
attention's splits inside the projection to values), 16 and 40 heads (one and two tiles of rows), contexts of one to nine splits, with
fewer and more than four beside one another, sequences whose newest entry opens a page, and prompts for the forms of the convolution."""
import numpy as np
import pytest

import jasmine_b200 as jb
import zugolorn_oracle as zo
import zugolorn_util as zu

pytestmark = pytest.mark.gpu
TOL = 0.08  # bf16 models (test_gpu_zugolorn.py)


@pytest.mark.parametrize("heads,batch", [(16, 1), (16, 8), (16, 9), (16, 17), (40, 3), (3, 16)])
def test_latent_attention_steps(heads, batch):
    cfg = zu.config([zu.attention(heads=heads, dim=40, rot_dim=16, vdim=24, kv_rank=72, window=300)], width=64)
    w = zu.random_weights(cfg, heads + batch)
    lens = [(1, 62, 63, 64, 127, 250, 330, 400)[b % 8] + b // 8 for b in range(batch)]
    seqs = [zu.tokens(n + 4, cfg["vocab"], 7 * n + b) for b, n in enumerate(lens)]
    want = [zo.forward(cfg, zu.oracle_weights(w), s)[-4:] for s in seqs]
    m = zu.build(cfg, w, "bfloat16", max_batch=batch, max_context=512, max_step_tokens=2048)
    rows = [m.open() for _ in seqs]
    for r, s, n in zip(rows, seqs, lens):
        m.step([(r, s[:n])], [n - 1])
    nxt, lg = np.empty(batch, np.int32), np.empty((batch, cfg["vocab"]), np.float32)
    for k in range(4):
        m.step_active(np.array([s[n + k] for s, n in zip(seqs, lens)], np.int32), nxt, lg)
        for b in range(batch):
            assert zu.error(lg[b:b + 1], want[b][k:k + 1]) < TOL, (b, lens[b], k)
        assert np.array_equal(nxt, lg.argmax(1))
    jb.check_device_errors()
    m.close()


@pytest.mark.parametrize("heads,batch,context", [(16, 3, 1100), (16, 9, 1100), (16, 16, 1100), (40, 5, 1100), (16, 1, 4160), (3, 2, 4160)])
def test_latent_attention_steps_of_many_splits(heads, batch, context):
    """Up to nine splits of two pages and more for tokens of both groups of eight, next to tokens of one to four; 33 splits and more of a long context (the merge's
    weights are formed in groups of 32).  The oracle's logits of the last tokens, whose keys are the whole window."""
    window = context - 60
    cfg = zu.config([zu.attention(heads=heads, dim=40, rot_dim=16, vdim=24, kv_rank=72, window=window)], width=64)
    w = zu.random_weights(cfg, heads * batch)
    longest = context - 8
    lens = [(longest, 70, 130, longest // 2, 257, 63, longest - 65, 520)[b % 8] - b // 8 for b in range(batch)]
    seqs = [zu.tokens(n + 3, cfg["vocab"], 11 * n + b) for b, n in enumerate(lens)]
    want = [zo.forward(cfg, zu.oracle_weights(w), s)[-3:] for s in seqs]
    m = zu.build(cfg, w, "bfloat16", max_batch=batch, max_context=context, max_step_tokens=2048)
    rows = [m.open() for _ in seqs]
    for r, s, n in zip(rows, seqs, lens):
        m.step([(r, s[:n])], [n - 1])
    nxt, lg = np.empty(batch, np.int32), np.empty((batch, cfg["vocab"]), np.float32)
    for k in range(3):
        m.step_active(np.array([s[n + k] for s, n in zip(seqs, lens)], np.int32), nxt, lg)
        for b in range(batch):
            assert zu.error(lg[b:b + 1], want[b][k:k + 1]) < TOL, (b, lens[b], k)
    jb.check_device_errors()
    m.close()


@pytest.mark.parametrize("dtype,tol", [("float32", 4e-5), ("bfloat16", TOL)])
@pytest.mark.parametrize("conv", [1, 3, 4, 6])
@pytest.mark.parametrize("inner,lens", [(48, [37]), (2400, [800, 803, 5, 796])])
def test_convolution_of_prompts(inner, lens, conv, dtype, tol):
    """Two and eight tokens per thread (the wide case has enough threads for eight), segments that end inside a thread's tokens."""
    cfg = zu.config([zu.mamba(inner=inner, state=4, conv=conv)], width=48)
    w = zu.random_weights(cfg, inner + conv)
    seqs = [zu.tokens(n, cfg["vocab"], n) for n in lens]
    m = zu.build(cfg, w, dtype, max_batch=len(lens), max_step_tokens=4096)
    rows, ends = [m.open() for _ in seqs], np.cumsum(lens)
    places = sorted({int(e) - 1 - k for e, n in zip(ends, lens) for k in (0, 1, min(n, 9) - 1)})
    _, lg = m.step(list(zip(rows, seqs)), places)
    want = np.concatenate([zo.forward(cfg, zu.oracle_weights(w), s) for s in seqs])[places]
    assert zu.error(lg, want) < tol
    m.close()


@pytest.mark.parametrize("rows,pitch,vocab,cap", [(1, 7, 7, 0.0), (3, 72, 70, 5.0), (2, 1001, 999, 3.0), (5, 32000, 32000, 30.0), (2, 70004, 70001, 0.0)])
def test_logits_and_their_maximum(rows, pitch, vocab, cap):
    """Rows of aligned fours and others, vocabularies that end inside a four, more logits than a thread holds at once, equal maxima, a padding that must not win."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = 4 * torch.randn(rows, pitch, generator=g, device="cuda")
    x[0, vocab // 2] = x[0, vocab - 1] = 100.0
    x[:, vocab:] = 1e6
    want = cap * torch.tanh(x.double() / cap) if cap else x.double()
    want[:, vocab:] = x[:, vocab:].double()
    nxt = jb.logits_finish(x, vocab, cap)
    assert torch.allclose(x.double(), want, rtol=1e-6, atol=1e-6)
    assert nxt.tolist() == x[:, :vocab].cpu().numpy().argmax(1).tolist() and nxt[0] == vocab // 2


@pytest.mark.parametrize("rows,pitch,vocab,cap", [(1, 4, 1, 2.0), (3, 72, 70, 5.0), (2, 8196, 8193, 0.0), (2, 8196, 8195, 3.0)])
def test_logits_whose_last_row_has_no_padding(rows, pitch, vocab, cap):
    """Rows of aligned fours in an allocation that ends with the last row's vocabulary (what lies behind it is not the caller's: nothing there is read)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = 4 * torch.randn((rows - 1) * pitch + vocab, generator=g, device="cuda")
    valid = torch.cat([torch.arange(vocab) + r * pitch for r in range(rows)]).cuda()
    before = x.clone()
    want = before[valid].reshape(rows, vocab).double()
    want = cap * torch.tanh(want / cap) if cap else want
    keys, ctrs, nxt = torch.zeros(rows, dtype=torch.int64, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.empty(rows, dtype=torch.int32, device="cuda")
    jb.check(jb.lib().jsm_logits_finish(x.data_ptr(), pitch, rows, vocab, cap, keys.data_ptr(), ctrs.data_ptr(), nxt.data_ptr(), jb.stream_ptr()))
    got = x[valid].reshape(rows, vocab)
    assert torch.allclose(got.double(), want, rtol=1e-6, atol=1e-6)
    assert nxt.tolist() == got.argmax(1).tolist()
    padding = torch.ones_like(x, dtype=torch.bool).index_fill(0, valid, False)
    assert torch.equal(x[padding], before[padding])
