"""Rotation and append of a prompt's fused rows in one pass: what the cache holds behind a prompt carries the next token like a prompt one token
longer, to the accuracy of two bf16 evaluations; and, with projections that are exact whatever the order of their sums, it holds the very bits that decode
steps append token by token, so that a key or value in a wrong place or rotated by a wrong angle shows (pages crossed and not, one and several query heads per
kv head, head counts that do and do not fill a pass over 64 heads)."""
import pytest
import torch

from jasmine_b200.model import Llama

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv", [(1, 1), (8, 2), (24, 24)])
@pytest.mark.parametrize("T", [2, 64, 65, 130])
def test_prompt_then_step_equals_longer_prompt(heads, kv, T):
    m = Llama(1, heads * 128, heads, kv, 256, 500, max_batch=2, max_context=192, seed=heads)
    ids = torch.randint(0, 500, (T,), generator=torch.Generator(device="cuda").manual_seed(T), device="cuda", dtype=torch.int32)
    nxt, whole, step = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.empty(500, device="cuda"), torch.empty(2, 500, device="cuda")
    m.prefill(ids, 0, nxt, whole)
    m.reset()
    for row in range(2):
        m.prefill(ids[:-1].contiguous(), row, nxt)
    m.decode_step(ids[-1:].repeat(2).contiguous(), nxt, step)
    # two bf16 evaluations with sums in another order, each held to 2e-2 of the oracle elsewhere
    assert float((step - whole).abs().max()) <= 4e-2 * float(whole.abs().max())
    m.close()


@pytest.mark.parametrize("heads,kv", [(1, 1), (8, 2), (24, 24)])
@pytest.mark.parametrize("T", [3, 64, 65, 130])
def test_prompt_leaves_the_bits_of_decode_steps(heads, kv, T):
    d = heads * 128
    g = torch.Generator(device="cuda").manual_seed(T)
    rows = (heads + 2 * kv) * 128
    w = torch.zeros(rows, d, device="cuda")  # one power of two per row: every projection is a single exact product
    w[torch.arange(rows, device="cuda"), torch.randint(0, d, (rows,), generator=g, device="cuda")] = \
        2.0 ** torch.randint(-1, 2, (rows,), generator=g, device="cuda") * (1 - 2 * torch.randint(0, 2, (rows,), generator=g, device="cuda"))
    ids = torch.randint(0, 500, (T,), generator=g, device="cuda", dtype=torch.int32)
    out = []
    for prompt in (T - 1, 1):
        m = Llama(1, d, heads, kv, 256, 500, max_batch=1, max_context=192, seed=heads)
        m.set_weight("layers.0.wqkv", w.bfloat16())
        nxt, logits = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(1, 500, device="cuda")
        m.prefill(ids[:prompt].contiguous(), 0, nxt)
        for t in range(prompt, T):
            m.decode_step(ids[t:t + 1].contiguous(), nxt, logits)
        out.append(logits.clone())
        m.close()
    assert torch.equal(out[0], out[1])
