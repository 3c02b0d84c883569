"""nn.Module whose call goes straight to ``forward`` when nothing else is registered.

A decode step calls half a dozen small modules per layer, each worth a few microseconds on the GPU; nn.Module's call path
(two Python frames, tracing and hook checks) is a third of their host time.
"""
from __future__ import annotations

import torch
from torch import nn
from torch.nn.modules import module as _torch_module

_GLOBAL_HOOKS = (_torch_module._global_forward_hooks, _torch_module._global_forward_pre_hooks,
                 _torch_module._global_backward_hooks, _torch_module._global_backward_pre_hooks)
_G0, _G1, _G2, _G3 = _GLOBAL_HOOKS                    # (torch keeps these dicts for the life of the process)
_module_call = nn.Module.__call__
_trace = torch.jit._trace                             # (its _trace_module_map is set while a trace names modules)


class DirectModule(nn.Module):
    def __call__(self, *args, **kwargs):
        d = self.__dict__
        if (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"]
                or _G0 or _G1 or _G2 or _G3 or self._compiled_call_impl is not None or _trace._trace_module_map is not None):
            return _module_call(self, *args, **kwargs)
        return self.forward(*args, **kwargs)
