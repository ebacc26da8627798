"""When a call may pass its operator by.

The library's adjoints are registered operators, so that traced and transformed
graphs see them; an operator call costs 100 to 150 us of host time on the Arm
host, most of a small step. A plain eager backward needs none of that and calls
the function behind the operator.
"""

from __future__ import annotations

import torch

_PLAIN = (torch.Tensor, torch.nn.Parameter)
_dispatch_modes = getattr(torch._C, "_len_torch_dispatch_stack", None)
_functorch = getattr(torch._C, "_functorch", None)
_interpreters = getattr(_functorch, "peek_interpreter_stack", None)
_legacy_batched = getattr(_functorch, "is_legacy_batchedtensor", None)


def plain_tensors(*tensors) -> bool:
    """Ordinary tensors (no fake, functional or other subclass, and not batched
    by the vmap of torch.autograd.grad(is_grads_batched=True), which enters no
    function transform) with no compiler, dispatch mode or function transform
    active: a launch may read their pointers. False where this torch cannot
    tell."""
    if torch.compiler.is_compiling():  # first: the compiler traces past it, not into the tests below
        return False
    if _dispatch_modes is None or _interpreters is None or _legacy_batched is None:
        return False
    if any(t is not None and (type(t) not in _PLAIN or _legacy_batched(t)) for t in tensors):
        return False
    return _dispatch_modes() == 0 and _interpreters() is None


def plain_eager(*tensors) -> bool:
    """Whether a backward may call the function behind its operator: plain
    tensors and no gradient recorded (a double backward must meet the operator,
    which refuses it)."""
    return not torch.is_grad_enabled() and plain_tensors(*tensors)
