"""The layers' short call path: whatever nn.Module's call path would run around forward still runs."""
import importlib

import pytest
import torch
from torch import nn
from torch.nn.modules import module as torch_module

module = importlib.import_module("nano-vllm-moe_b200.layers.module")


class Plain(nn.Module):
    def __init__(self):
        super().__init__()
        self.scale = nn.Parameter(torch.tensor(3.0))

    def forward(self, x, shift=0.0):
        return x * self.scale + shift


class Direct(module.DirectModule, Plain):
    pass


def record(register):
    """What a hook sees and returns on a plain module, and on a direct one."""
    seen = []
    for cls in (Plain, Direct):
        m, log = cls(), []
        handle = register(m, log)
        x = torch.tensor([1.0, 2.0], requires_grad=True)
        y = m(x, shift=0.5)
        y.sum().backward()
        handle.remove()
        m(x)                                           # removed hooks stay silent
        seen.append((log, y.detach().tolist(), x.grad.tolist(), m.scale.grad.item()))
    return seen


HOOKS = {
    "forward": lambda m, log: m.register_forward_hook(lambda mod, a, out: (log.append("f"), out * 2)[1]),
    "forward_kwargs": lambda m, log: m.register_forward_hook(lambda mod, a, kw, out: log.append(sorted(kw)), with_kwargs=True),
    "always_called": lambda m, log: m.register_forward_hook(lambda mod, a, out: log.append("a"), always_call=True),
    "forward_pre": lambda m, log: m.register_forward_pre_hook(lambda mod, a: (log.append("p"), (a[0] + 1,))[1]),
    "backward": lambda m, log: m.register_full_backward_hook(lambda mod, gi, go: (log.append("b"), (gi[0] * 4,))[1]),
    "backward_pre": lambda m, log: m.register_full_backward_pre_hook(lambda mod, go: (log.append("q"), (go[0] * 5,))[1]),
    "global_forward": lambda m, log: torch_module.register_module_forward_hook(lambda mod, a, out: (log.append("g"), out + 7)[1]),
    "global_forward_pre": lambda m, log: torch_module.register_module_forward_pre_hook(lambda mod, a: log.append("h")),
    "global_backward": lambda m, log: torch_module.register_module_full_backward_hook(lambda mod, gi, go: log.append("i")),
    "global_backward_pre": lambda m, log: torch_module.register_module_full_backward_pre_hook(lambda mod, go: log.append("j")),
}


@pytest.mark.parametrize("hook", list(HOOKS))
def test_hooks_run_as_on_any_module(hook):
    plain, direct = record(HOOKS[hook])
    assert plain[0] and plain == direct


def test_a_trace_keeps_the_modules_scopes():
    def scopes(cls):
        outer = nn.Sequential(cls(), cls())
        graph = torch.jit.trace(outer, torch.ones(2)).inlined_graph
        return [n.scopeName().replace(cls.__name__, "M") for n in graph.nodes() if n.kind() == "aten::mul"]
    assert scopes(Direct) == scopes(Plain) and all(scopes(Plain))


def test_a_compiled_call_is_taken():
    m = Direct()
    m._compiled_call_impl = lambda *a, **kw: "compiled"
    assert m(torch.ones(2)) == "compiled"


def test_without_hooks_forward_is_called_directly(monkeypatch):
    m = Direct()
    monkeypatch.setattr(nn.Module, "_call_impl", lambda *a, **kw: pytest.fail("the long way"))
    assert m(torch.ones(2), shift=1.0).tolist() == [4.0, 4.0]
