"""How this library's autograd nodes are called.  Their kernels take 3 to 30 us, less than what one ``apply`` costs on the
host: a node with ``setup_context`` has its ``forward`` inspected on every call (the signature alone took about 35 of
130 us, measured in a sampling pass of the twelve-block denoiser, which makes 73 such calls)."""
from __future__ import annotations

import inspect

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
