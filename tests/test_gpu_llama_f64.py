"""LLaMA-shape steps and prompts against the same model in float64: the projections of a batch (clusters, few and many tiles, fused norms, residual
and row statistics) and of prompts so long that the row statistics come from tiles of 256 features."""
import pytest
import torch

import jasmine_b200 as jb
from jasmine_b200.model import Llama
from llama_f64 import Reference

pytestmark = pytest.mark.gpu

BAR = 2e-2  # of the largest logit: the bar of a bf16 decoder elsewhere


def close(got, want):
    return float((got.double() - want).abs().max()) <= BAR * float(want.abs().max())


@pytest.mark.parametrize("batch", [1, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("d,kv,ffn", [(512, 4, 1152), (1024, 2, 2176), (2048, 16, 5504)])
def test_steps_of_a_batch(d, kv, ffn, batch):
    vocab = 1000
    m = Llama(2, d, d // 128, kv, ffn, vocab, max_batch=batch, max_context=64, seed=7)
    ref = Reference(m, 2, d, d // 128, kv, ffn, vocab)
    g = torch.Generator(device="cuda").manual_seed(batch)
    ids = torch.randint(0, vocab, (batch, 9), generator=g, device="cuda", dtype=torch.int32)
    nxt, logits = torch.zeros(batch, dtype=torch.int32, device="cuda"), torch.empty(batch, vocab, device="cuda")
    for b in range(batch):
        m.prefill(ids[b, :8].contiguous(), b)
    m.decode_step(ids[:, 8].contiguous(), nxt, logits)
    jb.check_device_errors()
    for b in sorted({0, 1, batch // 2, batch - 1} & set(range(batch))):
        assert close(logits[b], ref.logits(ids[b]))
    m.close()


@pytest.fixture(scope="module", params=[(4096, 32), (3968, 31)], ids=["32 tiles", "31 tiles"])
def wide(request):
    d, heads = request.param
    m = Llama(2, d, heads, 1, 1024, 1000, max_batch=700, max_context=704, seed=9)
    yield m, Reference(m, 2, d, heads, 1, 1024, 1000)
    m.close()


# the last token in different warps of the pair of CTAs that write a tile's statistics; 200: tiles of 128 features
@pytest.mark.parametrize("T", [200, 513, 600, 641, 700])
def test_prompts_with_statistics_of_wide_tiles(wide, T):
    m, ref = wide
    ids = torch.randint(0, 1000, (T,), generator=torch.Generator(device="cuda").manual_seed(T), device="cuda", dtype=torch.int32)
    nxt, logits = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(1000, device="cuda")
    m.reset()
    m.prefill(ids, 0, nxt, logits)
    jb.check_device_errors()
    assert close(logits, ref.logits(ids))
