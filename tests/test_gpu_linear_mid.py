"""The projection kernel for a few dozen tokens (and for few tokens and few tiles) over packed weights against float64 products of the same bf16 inputs: both edges of
its token blocks of 16 / 32 / 64 / 128, tiles and half tiles, one to eight CTAs per tile, k-blocks that do not divide among them, more
tiles than the chip holds at once, and the fused norm, residual and row statistics of a decoder step."""
import pytest
import torch

import jasmine_b200 as jb
import test_gpu_linear_tiled as tiled
from jasmine_b200.model import Llama

pytestmark = pytest.mark.gpu

SHAPES = [(1, 64, 64), (5, 160, 4096), (8, 2048, 2048), (9, 4100, 520), (16, 4096, 1032), (16, 2048, 5504), (17, 64, 64), (17, 132, 72), (31, 12, 2048), (32, 2048, 2048), (33, 388, 648), (40, 200, 4104), (63, 1000, 520), (64, 2048, 5504), (64, 6144, 2048),
          (64, 19204, 264), (65, 128, 4096), (100, 300, 4104), (127, 2048, 5504), (128, 4608, 4096)]


@pytest.mark.parametrize("T,N,K", SHAPES)
def test_plain_bias_activation_and_residual(T, N, K):
    tiled.test_plain_bias_activation_and_residual(T, N, K)


@pytest.mark.parametrize("T,N,K", SHAPES)
def test_gate_up_pairs(T, N, K):
    tiled.test_gate_up_pairs(T, N, K)


@pytest.mark.parametrize("batch", [9, 17, 33, 64])
@pytest.mark.parametrize("width,kv", [(512, 4), (1024, 2)])
def test_decoder_step_rows_agree_with_single_sequences(batch, width, kv):
    """A step of `batch` sequences (fused norms, residual, statistics) gives every row what it gets in a batch of its own."""
    make = lambda n: Llama(2, width, width // 128, kv, 2 * width + 128, 1000, max_batch=n, max_context=64, seed=7)  # noqa: E731
    m, one = make(batch), make(1)
    g = torch.Generator(device="cuda").manual_seed(batch)
    ids = torch.randint(0, 1000, (batch, 9), generator=g, device="cuda", dtype=torch.int32)
    nxt, logits = torch.zeros(batch, dtype=torch.int32, device="cuda"), torch.empty(batch, 1000, device="cuda")
    for b in range(batch):
        m.prefill(ids[b, :8].contiguous(), b, nxt)
    m.decode_step(ids[:, 8].contiguous(), nxt, logits)
    n1, l1 = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(1, 1000, device="cuda")
    for b in (0, 1, batch // 2, batch - 1):
        one.reset()
        one.prefill(ids[b, :8].contiguous(), 0, n1)
        one.decode_step(ids[b, 8:9].contiguous(), n1, l1)
        # two bf16 evaluations with sums in another order, each held to 2e-2 of the oracle elsewhere
        assert float((logits[b] - l1[0]).abs().max()) <= 4e-2 * float(l1.abs().max())
    jb.check_device_errors()
    m.close(), one.close()
