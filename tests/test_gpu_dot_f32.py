"""fp32 products at the edges of their tiles: the reference's order bit for bit (16 x 16 and 64 x 64 tiles, 16- and 4-byte copies),
and the products of fp32 models (16- and 64-row tiles, shared by clusters) against float64."""
import numpy as np
import pytest
import torch

import cases
import jasmine_b200 as jb
import oracle_lib as ol
import vagonex_oracle as vo
import vagonex_util as vu
from gpu_util import assert_close, dev, host

pytestmark = pytest.mark.gpu
port = ol.port_oracle()


# one row or column, remainders of the tiles and of blocks of 32 products, fewer and more blocks than the ring has stages, both tile sizes
@pytest.mark.parametrize("M,K,N", [(1, 33, 130), (17, 31, 15), (16, 32, 16), (33, 260, 31), (15, 1, 40), (700, 40, 450), (513, 67, 641), (64, 300, 4800)])
@pytest.mark.parametrize("layout", ["rows", "columns", "windows", "unaligned"])
def test_reference_order(M, K, N, layout):
    A, B = cases.normal((M, K), 420, M), cases.normal((K, N), 421, N)
    a, b, out = dev(A), dev(B), torch.empty(M, N, device="cuda")
    if layout == "columns":  # products contiguous in B, not in A
        a, b = a.t().contiguous().t(), b.t().contiguous().t()
    elif layout == "windows":  # contiguous products in both, 16-byte aligned rows of a wider matrix where 4 divides it
        pad = -K % 4 + 4
        wa, wb = torch.full((M, K + pad), torch.nan, device="cuda"), torch.full((N, K + pad), torch.nan, device="cuda")
        wa[:, :K], wb[:, :K] = a, b.t()
        a, b = wa[:, :K], wb[:, :K].t()
    elif layout == "unaligned":
        wa, wb = torch.full((M, K + 4), torch.nan, device="cuda"), torch.full((N, K + 3), torch.nan, device="cuda")
        wa[:, 1:K + 1], wb[:, :K] = a, b.t()
        a, b = wa[:, 1:K + 1], wb[:, :K].t()
    bias = torch.linspace(-1, 1, N, device="cuda")[None]
    jb.dot_f32(a, b, out, bias=bias, epilogue=1)
    rc, want = port.dot(A, B)
    want = want + host(bias)
    assert rc == 0 and np.array_equal(host(out), np.where(want > 0, want, 0 * want))


@pytest.fixture(scope="module")
def wide_model():
    cfg = vu.config([vu.lightning(heads=2, dim=36, vdim=40, ff=1100)], width=520, vocab=300)
    w = vu.random_weights(cfg, 31)
    toks = vu.tokens(160, cfg["vocab"], 32)
    m = vu.build(cfg, w)
    yield m, toks, vo.forward(cfg, vu.oracle_weights(w), toks)
    m.close()


@pytest.mark.parametrize("size", [1, 8, 16, 17, 32, 33, 64, 65, 160])
def test_products_of_fp32_models(wide_model, size):
    m, toks, want = wide_model
    assert_close(vu.run_portions(m, toks, [size]), want, 4e-5)  # (the bar of the other fp32 models)
