"""How this library's autograd nodes are called.  Their kernels take 3 to 30 us, less than what one ``apply`` costs on the
host: a node with ``setup_context`` has its ``forward`` inspected on every call (the signature alone took about 35 of
130 us, measured in a sampling pass of the twelve-block denoiser, which makes 73 such calls)."""
from __future__ import annotations

import importlib
import inspect
import warnings

import torch
import torch.autograd.forward_ad as fwAD


def node(cls):
    """Class decorator: ``inspect.signature(cls.forward)`` is worked out once instead of on every call."""
    cls.forward.__signature__ = inspect.signature(cls.forward)
    return cls


def unrecorded() -> bool:
    """Nothing can come of a node: gradients are off, no forward-mode level is open, no function transform is active and
    nothing is being traced (``torch.jit.trace`` records a node as one operation; of a bare ``forward`` it would see the
    allocations only, and the traced function would return them unwritten).  A node's ``forward`` may then be called
    directly (a sampling pass: 10.1 -> 6.4 ms with both)."""
    return (not torch.is_grad_enabled() and fwAD._current_level < 0 and not torch._C._are_functorch_transforms_active()
            and not torch.compiler.is_compiling() and not torch.jit.is_tracing())


def apply(cls, *args):
    """``cls.apply(*args)`` for a node whose ``forward`` takes no context, without the node where none can be recorded."""
    return cls.forward(*args) if unrecorded() else cls.apply(*args)


_module = None  # the compiled module; False where there is none for this torch


def _load():
    global _module
    from . import _lib, functional

    _lib.load()  # says how to build what is missing
    if not _lib.native_built():
        warnings.warn(f"{_lib.NATIVE_PATH} is missing or was compiled against another torch than {torch.__version__}: the ops run through "
                      "their classes in Python, whose calls take three times as long on the host.  Build it with "
                      "`python -c 'import __graft_entry__ as g; g.build()'` (or semicat_b200._lib.build_native()).", RuntimeWarning, stacklevel=3)
        _module = False
        return False
    mod = importlib.import_module("semicat_b200._native")
    mod.set_kernels(functional._kernels)
    _module = mod
    return mod


def set_kernels(kind: int) -> None:
    if _module:
        _module.set_kernels(kind)


def module():
    """The compiled module (loaded on first use; CUDA only), or ``False``."""
    return _load() if _module is None else _module


def native(name: str, first: torch.Tensor, *args):
    """Op ``name`` of ``csrc/torch_nodes.cpp`` on these arguments, or ``None`` where the situation or the inputs are none of
    its own: outside all function transforms, or inside one ``torch.func.jvp`` and nothing else, on plain CUDA tensors, with the
    module built.
    (One attention call under ``torch.func.jvp`` with its gradients: 780-850 us through the classes here, 230-260 us so; a sampling pass of the
    twelve-block denoiser 6.7 -> 3.7 ms.)"""
    if not first.is_cuda or torch.compiler.is_compiling():
        return None
    jvp = torch._C._are_functorch_transforms_active()
    if jvp:
        levels = torch._C._functorch.get_interpreter_stack()
        if len(levels) != 1 or levels[0].key() != torch._C._functorch.TransformType.Jvp:
            return None
    mod = _load() if _module is None else _module
    return getattr(mod, name)(jvp, first, *args) if mod else None
