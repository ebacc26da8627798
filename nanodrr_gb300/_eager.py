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
_interpreters = getattr(getattr(torch._C, "_functorch", None), "peek_interpreter_stack", None)
_key_included = getattr(torch._C, "_dispatch_tls_is_dispatch_key_included", None)
try:
    # Set while torch.autograd.grad(is_grads_batched=True) batches, which enters
    # no function transform. One question per call: asking each tensor whether
    # it is batched (is_legacy_batchedtensor) took 5 % of a small step.
    _LEGACY_VMAP = torch._C._parse_dispatch_key("VmapMode")
    _key_included(_LEGACY_VMAP)
except Exception:  # not in this torch
    _LEGACY_VMAP = None


def plain_tensors(*tensors) -> bool:
    """Ordinary tensors (no fake, functional or other subclass) with no
    compiler, dispatch mode, function transform or batching active: a launch may
    read their pointers. False where this torch cannot tell."""
    if torch.compiler.is_compiling():  # first: the compiler traces past it, not into the tests below
        return False
    if _dispatch_modes is None or _interpreters is None or _LEGACY_VMAP is None:
        return False
    for t in tensors:
        if type(t) not in _PLAIN and t is not None:
            return False
    return _dispatch_modes() == 0 and _interpreters() is None and not _key_included(_LEGACY_VMAP)


def plain_eager(*tensors) -> bool:
    """Whether a backward may call the function behind its operator: plain
    tensors and no gradient recorded (a double backward must meet the operator,
    which refuses it)."""
    return not torch.is_grad_enabled() and plain_tensors(*tensors)
