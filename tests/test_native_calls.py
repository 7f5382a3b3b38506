"""The extension module behind the frequent calls of the Python plumbing (csrc/py_calls.cpp): the same results, refusals and exceptions as through ctypes
for every form of operand, and nothing taken that is not a plain dense CUDA tensor."""
import sys

import numpy as np
import pytest
import torch

import jasmine_b200 as jb

LEAF = [(jb.OP_LEAF, 0)]


def test_what_it_leaves_to_the_python_code():
    m = jb._calls()
    assert m, "jasmine_b200/_native.so is not built"
    t = torch.zeros(4, 4)
    assert m.dot_f32(t, t, t, None, 0, None) is None  # host memory
    assert m.dot_f32(1, t, t, None, 0, None) is None and m.dot_f32(t, t) is None
    assert m.eval_rows(jb.ROWS_SUM, 1, LEAF, [t], t, None, None, 0.0) is None
    assert m.embedding(t, t, None, None, None) is None
    with pytest.raises(TypeError):
        m.bind()


def test_a_module_of_another_torch_is_not_used(monkeypatch):
    m = jb._calls()
    assert m.torch == f"{torch.__version__} {torch.version.git_version}"
    monkeypatch.setattr(jb, "_calls_module", None)
    monkeypatch.setattr(m, "torch", "1.0 0000")
    with pytest.warns(UserWarning, match="built for torch 1.0"):
        assert jb._calls() is False
    assert jb._calls() is False  # (asked once)


def test_a_module_that_does_not_load_is_said(monkeypatch):
    monkeypatch.setattr(jb, "_calls_module", None)
    monkeypatch.setitem(sys.modules, "jasmine_b200._native", None)
    with pytest.warns(UserWarning, match="does not load"):
        assert jb._calls() is False


def test_a_module_that_is_not_there_is_no_matter(monkeypatch, tmp_path, recwarn):
    monkeypatch.setattr(jb, "_calls_module", None)
    monkeypatch.setattr(jb, "PKG_DIR", tmp_path)
    assert jb._calls() is False and not recwarn.list


def both(monkeypatch, call):
    """Result or exception of call() through the module and through ctypes."""
    out = []
    for use in (jb._calls(), False):
        monkeypatch.setattr(jb, "_calls_module", use)
        if not use:
            monkeypatch.setattr(jb, "_calls", lambda: False)
        try:
            out.append(call())
        except Exception as e:  # noqa: BLE001
            out.append((type(e), str(e)))
    return out


@pytest.mark.gpu
def test_same_results_and_exceptions(monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(1)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    new = lambda r, c: torch.full((r, c), 7.0, device="cuda")  # noqa: E731
    a, b, bias, gain, wide = rn(6, 10), rn(10, 8), rn(1, 8), rn(10), rn(12, 40)
    ids, at = torch.tensor([3, 0, 5, 1], dtype=torch.int32, device="cuda"), torch.arange(4, dtype=torch.int32, device="cuda")
    grad = rn(6, 10).requires_grad_()
    q, k = rn(6, 64), rn(6, 32)
    axpb = [(jb.OP_LEAF, 0), (jb.OP_IMM, 2), (jb.OP_MUL,), (jb.OP_LEAF, np.int64(1)), (jb.OP_ADD,)]
    calls = [
        lambda: jb.dot_f32(a, b, new(6, 8)),
        lambda: jb.dot_f32(b.t(), a.t(), new(8, 6), epilogue=2),
        lambda: jb.dot_f32(wide[1:7, 3:33:3], b, new(6, 8), bias=bias, epilogue=3, residual=rn(1, 8).expand(6, 8) * 0 + 1),
        lambda: jb.dot_f32(a, b, new(8, 8)[1:7], bias=bias[0]),
        lambda: jb.dot_f32(grad, b, new(6, 8)).detach(),
        lambda: jb.dot_f32(torch.nn.Parameter(a), b, new(6, 8)),
        lambda: jb.dot_f32(a, a, new(6, 8)),                      # shapes that do not match
        lambda: jb.dot_f32(a.double(), b, new(6, 8)),             # a type without a place in a matrix
        lambda: jb.dot_f32(a.bfloat16(), b, new(6, 8)),           # one that the product refuses
        lambda: jb.dot_f32(a[None], b, new(6, 8)),                # three dimensions
        lambda: jb.dot_f32(a, b, new(6, 8), epilogue=9),
        lambda: jb.dot_f32(a[:0], b, new(0, 8)),
        lambda: torch.vmap(lambda x: jb.dot_f32(x, b, new(6, 8)))(a[None]),  # (no memory of its own: an exception either way)
        lambda: jb.eval_rows(jb.ROWS_LAYERNORM, 1, LEAF, [a], new(6, 10), gain=gain, bias=gain, eps=1e-5),
        lambda: jb.eval_rows(jb.ROWS_SUM, 0, LEAF, [wide.t()], new(1, 12)),
        lambda: jb.eval_rows(jb.ROWS_SOFTMAX, 1, axpb, [wide[:, :10], gain], new(12, 10)),
        lambda: jb.eval_rows(jb.ROWS_ARGMAX, 1, LEAF, [a], torch.zeros(6, 1, dtype=torch.int32, device="cuda")),
        lambda: jb.eval_rows(99, 1, LEAF, [a], new(6, 10)),
        lambda: jb.eval_elementwise(axpb, [a, a], new(6, 10)),
        lambda: jb.eval_elementwise([(jb.OP_LEAF, 0), (jb.OP_POW, 3.0)], (a,), new(6, 10)),
        lambda: jb.eval_elementwise([(jb.OP_LEAF, 1)], [a], new(6, 10)),  # a leaf that is not there
        lambda: jb.eval_elementwise(LEAF * 40, [a], new(6, 10)),          # a program too long
        lambda: jb.embedding(wide, ids),
        lambda: jb.embedding(wide, ids, rn(4, 40) * 0 + 1, at),
        lambda: jb.embedding(wide[:, :39].contiguous(), ids),             # rows that are no whole vectors
        lambda: jb.attn_prefill(q, k, k, 2, 4, 2, 16),
        lambda: jb.attn_prefill(q, k, k, 1, 4, 2, 16, causal=False, scale=1),
        lambda: jb.attn_prefill(q, k, k, 0, 4, 2, 16),                    # no sequences
    ]
    for i, call in enumerate(calls):
        torch.manual_seed(i)
        g.manual_seed(i)
        x, y = None, None
        results = []
        for r in both(monkeypatch, lambda: (g.manual_seed(i), call())[1]):
            results.append(r)
        x, y = results
        if isinstance(x, tuple) or isinstance(y, tuple):
            assert x == y, (i, x, y)
        else:
            assert torch.equal(x, y), i
        monkeypatch.undo()
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_the_current_stream_is_taken():
    a, b, out = torch.randn(64, 64, device="cuda"), torch.randn(64, 64, device="cuda"), torch.zeros(64, 64, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):  # a launch on any other stream would end the capture with an error
            jb.dot_f32(a, b, out)
    assert not out.any()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.allclose(out, a @ b, atol=1e-3)


@pytest.mark.gpu
def test_a_tensor_that_keeps_its_address_raises():
    """An exception of torch inside the module is the Python code's to raise, not the end of the process."""
    closed = torch.randn(8, 8, device="cuda")
    torch._C._set_throw_on_mutable_data_ptr(closed)
    a, out, ids = torch.randn(8, 8, device="cuda"), torch.empty(8, 8, device="cuda"), torch.zeros(8, dtype=torch.int32, device="cuda")
    for call in (lambda: jb.dot_f32(a, closed, out), lambda: jb.dot_f32(closed, a, out), lambda: jb.eval_elementwise(LEAF, [closed], out),
                 lambda: jb.eval_rows(jb.ROWS_SOFTMAX, 1, LEAF, [a], closed), lambda: jb.embedding(closed, ids), lambda: jb.attn_prefill(closed, a, a, 1, 1, 1, 8)):
        with pytest.raises(RuntimeError, match="data pointer"):
            call()
    assert torch.allclose(jb.dot_f32(a, a, out), a @ a, atol=1e-4)
