"""Projections that stay with the streaming kernel beyond 16 tokens: more packed tiles of 128 rows than the chip has multiprocessors (17 to 64
tokens), deep ones whose tiles cover them, deep or wide matrices up to 128 tokens, very deep ones of a few tiles up to 256, and shallow ones of few blocks of depth."""
import pytest
import torch

import jasmine_b200 as jb
import test_gpu_linear_tiled as tiled
from jasmine_b200.model import Llama
from llama_f64 import Reference
from test_gpu_trace import traced

pytestmark = pytest.mark.gpu

# both edges of the token blocks of 32 / 64 / 128 / 256, ragged last tiles and blocks of depth
SHAPES = [(17, 4096, 4096), (32, 4100, 4104), (33, 4096, 4352), (64, 4700, 4104), (31, 11400, 4096), (64, 12288, 4104), (17, 19204, 520), (32, 19076, 1032), (33, 20000, 520), (64, 18948, 1096), (24, 8192, 256), (16, 4100, 200), (65, 9604, 4104), (96, 9600, 4096),
          (80, 19204, 4104), (128, 37892, 4104), (128, 11400, 8200), (80, 5892, 8200), (129, 292, 8200), (256, 1000, 8264)]
PAIRS = [(17, 2048, 4096), (32, 2052, 4104), (64, 2300, 4160), (48, 6000, 4096), (17, 9604, 520), (32, 9540, 1032), (33, 10000, 520), (64, 9476, 1096), (16, 1028, 200), (65, 4804, 4104), (80, 9604, 4104), (128, 18948, 4104),
         (160, 292, 8200)]


@pytest.mark.parametrize("T,N,K", SHAPES)
def test_plain_bias_activation_and_residual(T, N, K):
    tiled.test_plain_bias_activation_and_residual(T, N, K)


@pytest.mark.parametrize("T,N,K", PAIRS)
def test_gate_up_pairs(T, N, K):
    tiled.test_gate_up_pairs(T, N, K)


@pytest.mark.parametrize("T", [17, 32, 64, 80])
def test_more_tiles_than_multiprocessors_are_split_evenly(T):
    """172 tiles: a launch of a CTA per tile would leave most SMs idle while the last 24 tiles run alone."""
    N, K = 11008, 4096
    X, W = tiled.inputs(T, 2 * N, K, 3)
    Wp = jb.linear_pack(W, N, paired=True)
    out = torch.empty(T, N, device="cuda", dtype=torch.bfloat16)
    (rec,) = traced(lambda: jb.linear_bf16_packed(X, Wp, out, epilogue=3))
    sms = rec.shape[0]
    if 2 * N // 128 <= sms:
        pytest.skip("a chip with an SM for every tile")
    assert int((rec[:, 0] > 0).sum()) == sms
    assert int((rec[:, 6] > 0).sum()) > sms // 2  # most CTAs end a second piece of the stream


@pytest.mark.parametrize("d,kv,ffn,batch", [(1024, 8, 9600, 17), (1024, 2, 9608, 64), (512, 4, 9608, 32), (2048, 4, 11008, 33), (4096, 32, 1024, 17), (4096, 32, 1024, 40), (4096, 4, 4608, 64)])
def test_batched_steps_of_wide_projections(d, kv, ffn, batch):
    """A step with the fused norm in front of a gate/up projection and a vocabulary of more tiles than SMs, or with the projections of the 7B width."""
    vocab = 19100 if d < 4096 else 1000
    m = Llama(1, d, d // 128, kv, ffn, vocab, max_batch=batch, max_context=64, seed=11)
    ref = Reference(m, 1, d, d // 128, kv, ffn, vocab)
    g = torch.Generator(device="cuda").manual_seed(batch)
    ids = torch.randint(0, vocab, (batch, 7), generator=g, device="cuda", dtype=torch.int32)
    nxt, logits = torch.zeros(batch, dtype=torch.int32, device="cuda"), torch.empty(batch, vocab, device="cuda")
    for b in range(batch):
        m.prefill(ids[b, :6].contiguous(), b)
    m.decode_step(ids[:, 6].contiguous(), nxt, logits)
    jb.check_device_errors()
    for b in (0, 1, batch // 2, batch - 1):
        want = ref.logits(ids[b])
        assert float((logits[b].double() - want).abs().max()) <= 2e-2 * float(want.abs().max())
    m.close()
