"""Whether a module's ``forward`` is the one of its class, with nobody looking on: fused paths that pass modules by ask first."""
from __future__ import annotations

from torch.nn.modules import module as _torch


def unobserved(*modules, backward: bool = False) -> bool:
    """True when no hook (of a module or of all of them) sees or changes what goes into or comes out of ``modules`` and none
    has a ``forward`` of its own set on the instance.  ``backward``: nor their gradients."""
    if _torch._global_forward_hooks or _torch._global_forward_pre_hooks:
        return False
    if backward and (_torch._global_backward_hooks or _torch._global_backward_pre_hooks):
        return False
    return not any(m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__
                   or (backward and (m._backward_hooks or m._backward_pre_hooks)) for m in modules)
