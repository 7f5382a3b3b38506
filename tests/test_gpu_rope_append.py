"""Rotation and append of a prompt's fused rows in one pass: what the cache holds behind a prompt must carry the next token exactly as
if the prompt had been one token longer (pages crossed and not, one and several query heads per kv head, head counts that do and do
not fill a pass over 64 heads)."""
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
