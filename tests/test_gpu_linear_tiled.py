"""The tiled projection kernel (calls of many tokens over packed weights) against float64 products of the same bf16 inputs, at the
edges of its tiles: token blocks of 256 (128 per CTA), feature tiles of 64 / 128 / 256, k-blocks of 64 taken two at a time."""
import pytest
import torch

import jasmine_b200 as jb

pytestmark = pytest.mark.gpu

# tokens, features, depth: below / at / above a token block, ragged last feature tile, odd number of packed tiles, odd number of
# k-blocks, a last k-block of 8, every tile width, more tiles than clusters
SHAPES = [(65, 64, 64), (100, 132, 72), (128, 260, 200), (129, 128, 128), (255, 384, 1032), (256, 1000, 520), (257, 640, 4096), (300, 388, 648),
          (513, 12, 2048), (1000, 4096, 576), (1025, 9600, 264), (2047, 6144, 1024)]


def bound(X, W, K, bf16_out, want):
    """fp32 sums that may truncate at every accumulated block of 16 products, then one rounding to bf16."""
    terms = (K + 15) // 16 + 16
    e = terms * 2.0 ** -23 * (X.abs().double() @ W.abs().double().t())
    return e + want.abs() * 2.0 ** -8 if bf16_out else e


def inputs(T, N, K, seed):
    X, W = (torch.empty(s, device="cuda", dtype=torch.bfloat16) for s in ((T, K), (N, K)))
    jb.fill(X, seed, 0, 0, 0.0, 1.0)
    jb.fill(W, seed, 1, 0, 0.0, 0.05)
    return X, W


@pytest.mark.parametrize("T,N,K", SHAPES)
def test_plain_bias_activation_and_residual(T, N, K):
    X, W = inputs(T, N, K, 500 + T)
    Wp = jb.linear_pack(W, N)
    bias = torch.empty(N, device="cuda"); jb.fill(bias, 1, 2, 0, 0.0, 1.0)
    R = torch.empty(T, N, device="cuda", dtype=torch.bfloat16); jb.fill(R, 1, 3, 0, 0.0, 1.0)
    base = X.double() @ W.double().t()
    for dtype in (torch.float32, torch.bfloat16):
        for epilogue, b, want in ((0, None, base), (1, bias, torch.relu(base + bias.double())), (2, bias, torch.nn.functional.gelu(base + bias.double())),
                                  (4, None, base + R.double())):
            out = torch.full((T + 1, N), 7.0, device="cuda", dtype=dtype)
            if epilogue == 4 and dtype == torch.bfloat16:  # the residual stream is updated in place
                out[:T] = R
                jb.linear_bf16_packed(X, Wp, out[:T], epilogue=4, residual=out[:T])
            else:
                jb.linear_bf16_packed(X, Wp, out[:T], bias=b, epilogue=epilogue, residual=R if epilogue == 4 else None)
            jb.check_device_errors()
            tol = bound(X, W, K, dtype == torch.bfloat16, want) * 1.2 + 2.0 ** -21 * (1.0 + want.abs())  # (gelu' < 1.13; adds in fp32)
            assert bool(((out[:T].double() - want).abs() <= tol).all()), (dtype, epilogue)
            assert bool((out[T] == 7.0).all()), "a row behind the last token was written"
    again = torch.empty(T, N, device="cuda", dtype=torch.float32)
    first = torch.empty_like(again)
    jb.linear_bf16_packed(X, Wp, first)
    jb.linear_bf16_packed(X, Wp, again, chained=True)
    assert torch.equal(first, again)


@pytest.mark.parametrize("T,N,K", SHAPES)
def test_gate_up_pairs(T, N, K):
    X, W = inputs(T, 2 * N, K, 600 + T)
    Wp = jb.linear_pack(W, N, paired=True)
    y = X.double() @ W.double().t()
    g, u = y[:, :N], y[:, N:]
    e = bound(X, W, K, False, y)
    eg, eu = e[:, :N], e[:, N:]
    gc, uc = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
    cases = {3: (torch.nn.functional.silu(g) * u, 1.1 * eg * (u.abs() + eu) + (g.abs() + eg) * eu),
             5: (gc * torch.sigmoid(1.702 * gc) * (uc + 1.0), 2.5 * 1.3 * eg + 1.5 * eu),
             6: (torch.nn.functional.gelu(g, approximate="tanh") * u, 1.13 * eg * (u.abs() + eu) + (g.abs() + eg) * eu)}
    for epilogue, (want, err) in cases.items():
        out = torch.full((T + 1, N), 7.0, device="cuda", dtype=torch.bfloat16)
        if epilogue == 5:
            jb.linear_bf16_packed_glu(X, Wp, out[:T], 1.702, 1.5)
        else:
            jb.linear_bf16_packed(X, Wp, out[:T], epilogue=epilogue)
        jb.check_device_errors()
        # the activation in fp32 with the 2-ulp division and the fast exponential (2 + |x| 2^-22 relative ulps), then bf16
        tol = err + want.abs() * (2.0 ** -8 + 2.0 ** -18) + 2.0 ** -20
        assert bool(((out[:T].double() - want).abs() <= tol).all()), epilogue
        assert bool((out[T] == 7.0).all())
