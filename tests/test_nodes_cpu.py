"""When the library's autograd nodes may be left out: only where nothing could be recorded."""
import inspect
import types
import warnings

import pytest
import torch
import torch.autograd.forward_ad as fwAD

from semicat_b200 import _lib, _nodes, dual_ops, functional, rotary


def test_unrecorded_only_without_gradients_transforms_and_forward_mode():
    assert not _nodes.unrecorded()
    with torch.no_grad():
        assert _nodes.unrecorded()
        with fwAD.dual_level():
            assert not _nodes.unrecorded()
        seen = []
        probe = lambda x: (seen.append(_nodes.unrecorded()), x * 2)[1]
        torch.func.jvp(probe, (torch.ones(2),), (torch.ones(2),))
        torch.func.vmap(probe)(torch.ones(2, 2))
        torch.func.grad(lambda x: probe(x).sum())(torch.ones(2))
        assert seen == [False] * 3
        with torch.enable_grad():
            assert not _nodes.unrecorded()
    with torch.inference_mode():
        assert _nodes.unrecorded()


def test_node_signatures_are_those_of_forward():
    nodes = [functional._AttentionDual, *(v for m in (dual_ops, rotary) for v in vars(m).values()
                                          if inspect.isclass(v) and issubclass(v, torch.autograd.Function))]
    assert len(nodes) > 8
    for cls in nodes:
        kept = cls.forward.__signature__
        del cls.forward.__signature__
        try:
            assert kept == inspect.signature(cls.forward)
        finally:
            cls.forward.__signature__ = kept


def test_apply_records_where_gradients_are_on():
    class Twice(torch.autograd.Function):
        @staticmethod
        def forward(x):
            return x * 2

        @staticmethod
        def setup_context(ctx, inputs, output):
            pass

        @staticmethod
        def backward(ctx, g):
            return g * 2

    _nodes.node(Twice)
    x = torch.ones(3, requires_grad=True)
    y = _nodes.apply(Twice, x)
    y.sum().backward()
    assert torch.equal(x.grad, torch.full((3,), 2.0))
    with torch.no_grad():
        z = _nodes.apply(Twice, x)
    assert torch.equal(z, y) and not z.requires_grad


class _Outside(torch.autograd.Function):
    """Doubles its input as a kernel does, where a tracer sees nothing of it but the allocation."""

    @staticmethod
    def forward(x):
        y = torch.empty_like(x)
        y.numpy()[...] = 2 * x.numpy()
        return y

    @staticmethod
    def setup_context(ctx, inputs, output):
        pass

    @staticmethod
    def backward(ctx, g):
        return g * 2


def test_a_trace_records_the_node():
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: _nodes.apply(_Outside, x) + 1, (torch.ones(3),), check_trace=False)
        assert torch.equal(traced(torch.full((3,), 5.0)), torch.full((3,), 11.0))
        seen = []
        torch.jit.trace(lambda x: (seen.append(_nodes.unrecorded()), x + 1)[1], (torch.ones(3),), check_trace=False)
        assert seen == [False]


def test_without_the_compiled_module_the_classes_run(monkeypatch, tmp_path):
    """Missing, or compiled against another torch: the native entries take no call, and say so once."""
    _lib.build()
    monkeypatch.setattr(_lib, "NATIVE_PATH", str(tmp_path / "_native.so"))
    monkeypatch.setattr(_lib, "NATIVE_TORCH_PATH", str(tmp_path / "_native.so.torch"))
    assert not _lib.native_built()
    (tmp_path / "_native.so").write_bytes(b"")
    assert _lib.native_built()
    (tmp_path / "_native.so.torch").write_text("1.0\n")
    assert not _lib.native_built()
    monkeypatch.setattr(_nodes, "_module", None)
    cuda = types.SimpleNamespace(is_cuda=True)
    with pytest.warns(RuntimeWarning, match="compiled against another torch"):
        assert _nodes.native("gelu", cuda) is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _nodes.native("gelu", cuda) is None and not _nodes.module()
        _nodes.set_kernels(0)
    (tmp_path / "_native.so.torch").write_text(torch.__version__ + "\n")
    assert _lib.native_built()
