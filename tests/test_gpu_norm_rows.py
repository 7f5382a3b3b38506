"""Norms of a sublayer's output around a token per multiprocessor, where the gain stops arriving ahead of the predecessor's end: models of both
norm places against their plain float64 implementations, and the operations at the remainders of a CTA's columns."""
import pytest
import torch

import jasmine_b200 as jb
import vagonex_oracle as vo
import vagonex_util as vu
import zugolorn_oracle as zo
import zugolorn_util as zu
from gpu_util import assert_close

pytestmark = pytest.mark.gpu


def portions():
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148
    return [sms, sms + 1, 7]


def test_norm_of_the_sum_in_a_model():
    cfg = vu.config([vu.lightning(heads=2, dim=20, vdim=24, ff=60), vu.attention(ff=52)], alpha=0.8)
    w, toks = vu.random_weights(cfg, 71), vu.tokens(sum(portions()), 72, 72)
    m = vu.build(cfg, w)
    assert_close(vu.run_portions(m, toks, portions()), vo.forward(cfg, vu.oracle_weights(w), toks), 4e-5)  # (the bar of the other fp32 models)
    m.close()


def test_norm_added_in_a_model():
    cfg = zu.config([zu.attention(ff=44), zu.mamba()])
    w, toks = zu.random_weights(cfg, 73), zu.tokens(sum(portions()), cfg["vocab"], 74)
    m = zu.build(cfg, w)
    assert_close(zu.run_portions(m, toks, portions()), zo.forward(cfg, zu.oracle_weights(w), toks), 4e-5)
    m.close()


@pytest.mark.parametrize("rows", [1, 149, 600])
@pytest.mark.parametrize("d", [8, 2048, 2056, 4096, 4104])
def test_operations(rows, d):
    g = torch.Generator(device="cuda").manual_seed(rows + d)
    y, x, gain = (torch.randn(s, generator=g, device="cuda") for s in ((rows, d), (rows, d), (d,)))
    for alpha in (None, 0.75):
        s = y.double() if alpha is None else alpha * x.double() + y.double()
        want = s * torch.rsqrt((s * s).mean(1, keepdim=True) + 1e-5) * gain.double() + (x.double() if alpha is None else 0.0)
        out, xb = x.clone(), torch.empty(rows, d, device="cuda", dtype=torch.bfloat16)
        jb.post_norm_add(y, out, gain, 1e-5, xb) if alpha is None else jb.sum_norm(y, out, gain, 1e-5, alpha, xb)
        # sums of at most 17 + 8 roundings per thread and tree, a division and a product
        assert bool(((out.double() - want).abs() <= 40 * 2.0 ** -24 * (want.abs() + x.abs().double() + 1e-3)).all())
        assert torch.equal(xb, out.bfloat16())
