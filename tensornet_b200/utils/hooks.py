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


def own_step(model, model_cls, sub_model, sub_cls) -> bool:
    """Whether a training step of ``model`` may pass by the calls of the model, of its dense part and of its ``Dense(1)`` head: they
    are the package's own (a subclass of the user's may add methods, not replace the ones passed by), on a GPU, with nobody looking on."""
    from ..core.runtime import runtime
    from ..layers.dense import DenseHead

    cls = type(model)
    if not runtime().on_gpu or type(sub_model) is not sub_cls or type(sub_model.head) is not DenseHead:
        return False
    if any(getattr(cls, k) is not getattr(model_cls, k) or k in model.__dict__ for k in ("forward", "__call__", "_loss")):
        return False
    return unobserved(model, sub_model, sub_model.head, backward=True)
