"""Whether a module may be passed by: fused paths that do a module's work without calling it, or call it with another layout, ask here."""
from __future__ import annotations

import torch.nn as nn
import torch.nn.modules.module as _m

_CALL = nn.Module.__call__


def observed(module, cls) -> bool:
    """True when calling ``module`` would run anything besides ``cls.own_forward``, the forward that class ``cls`` was written with: a
    subclass, a forward replaced on the class or the instance, or hooks on the module or on all modules."""
    return bool(type(module) is not cls or cls.forward is not cls.own_forward or cls.__call__ is not _CALL or "forward" in module.__dict__
                or module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks
                or _m._global_forward_hooks or _m._global_forward_pre_hooks or _m._global_backward_hooks or _m._global_backward_pre_hooks)
