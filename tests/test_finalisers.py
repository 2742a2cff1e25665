"""Objects of one reference cycle are finalised in any order (at interpreter
exit the modules' globals are such a cycle): a Langevin handle whose context
went first is not handed to the library, which would free its buffer on the
stream of a context that no longer exists."""
from __future__ import annotations

import pytest

import qew_gb300 as Q


class Lib:
    def __init__(self):
        self.calls = []

    def qew_ctx_destroy(self, h):
        self.calls.append("ctx")

    def qew_langevin_destroy(self, h):
        assert "ctx" not in self.calls
        self.calls.append("langevin")


@pytest.mark.parametrize("first", ["context", "dynamics"])
def test_dynamics_finalised_after_its_context(first):
    ctx = Q.Context.__new__(Q.Context)
    dyn = Q.LangevinDynamics.__new__(Q.LangevinDynamics)
    ctx.lib = lib = Lib()
    ctx.h, dyn.h, dyn.ctx = 1, 2, ctx
    for o in ((ctx, dyn) if first == "context" else (dyn, ctx)):
        o.__del__()
    assert lib.calls == (["ctx"] if first == "context" else ["langevin", "ctx"])
    assert ctx.h is None and dyn.h is None
