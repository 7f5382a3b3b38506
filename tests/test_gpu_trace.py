"""Time stamps of the projections (jsm_trace_begin / jsm_trace_end): one record per launch, whichever kernel runs it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYERS = 2


def traced(call, n_max=64):
    """Records [launches][CTAs][8] of what call() launches."""
    import torch

    import jasmine_b200 as jb
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    jb.check(jb.lib().jsm_trace_begin(n_max))
    call()
    torch.cuda.synchronize()
    buf, n, ctas = np.zeros((n_max, sms, 8), np.uint64), C.c_int(), C.c_int()
    jb.check(jb.lib().jsm_trace_end(buf.ctypes.data, n_max, C.byref(n), C.byref(ctas)))
    assert ctas.value == sms
    return buf[:n.value].astype(np.int64)


def check_records(t):
    last = 0
    for rec in t:
        rec = rec[rec[:, 0] > 0]
        assert len(rec), "a launch without stamps"
        resident, wait, first, mma, done = (rec[:, i] for i in (0, 2, 3, 4, 7))
        issued = mma > 0  # (of a pair of CTAs one issues the products)
        assert issued.any() and (resident <= wait).all() and (wait <= done).all()
        assert (first[issued] <= mma[issued]).all() and (mma[issued] <= done[issued]).all() and (rec[:, 5] <= done).all()
        assert done.max() >= last  # launches end in stream order
        last = done.max()


@pytest.mark.parametrize("batch", [1, 8, 17, 64])
def test_every_projection_of_a_step_is_recorded(batch):
    import torch

    from jasmine_b200.model import Llama
    m = Llama(LAYERS, 512, 4, 4, 1024, 1024, max_batch=batch, max_context=64, seed=3)
    ids = torch.arange(batch, dtype=torch.int32, device="cuda")
    nxt = torch.empty_like(ids)
    m.decode_step(ids, nxt)
    t = traced(lambda: m.decode_step(ids, nxt))
    m.close()
    assert len(t) == 4 * LAYERS + 1  # qkv, wo, gate/up, down of every layer, and the vocabulary
    check_records(t)


def test_every_projection_of_a_prompt_is_recorded():
    import torch

    from jasmine_b200.model import Llama
    m = Llama(LAYERS, 512, 4, 4, 1024, 1024, max_batch=1, max_context=256, seed=3)
    ids = torch.arange(200, dtype=torch.int32, device="cuda")
    nxt = torch.zeros(1, dtype=torch.int32, device="cuda")
    m.prefill(ids, 0, nxt)
    t = traced(lambda: m.prefill(ids, 0, nxt))
    m.close()
    assert len(t) == 4 * LAYERS + 1
    check_records(t)
