"""The two modules as a base class: overriding or wrapping ``block``, with the kernels' entry points replaced by a stub
(no GPU needed: what is checked is which Python code runs, how often, and with which tensors)."""

import pytest
import torch
import torch.nn.utils.parametrize

from miniworld_engine_b200 import BidirectionalTriangleMultiplicationB200, TriangleMultiplicationB200, bidirectional, functional

MODULES = {"single": TriangleMultiplicationB200, "bidirectional": BidirectionalTriangleMultiplicationB200}


@pytest.fixture
def calls(monkeypatch):
    """Keyword arguments of every call that would have gone to the kernels; the stub returns the pair tensor."""
    seen = []

    def stub(pair, mask=None, **kw):
        assert not torch.is_grad_enabled()
        seen.append(kw)
        return pair.detach().clone()

    monkeypatch.setattr(functional, "trimul_forward", stub)
    monkeypatch.setattr(bidirectional, "bidir_trimul_forward", stub)
    return seen


@pytest.mark.parametrize("grad", [True, False], ids=["grad", "no_grad"])
@pytest.mark.parametrize("base", MODULES.values(), ids=MODULES)
def test_an_override_of_block_runs_once(calls, base, grad):
    class Doubled(base):
        entered = 0

        def block(self, *args, **kwargs):
            self.entered += 1
            return 2 * super().block(*args, **kwargs)

    m, x = Doubled(8), torch.ones(1, 3, 3, 8)
    with torch.set_grad_enabled(grad):
        y = m.block(x)
        assert torch.is_grad_enabled() == grad
    assert m.entered == 1 and len(calls) == 1
    assert torch.equal(y, 2 * x)


@pytest.mark.parametrize("grad", [True, False], ids=["grad", "no_grad"])
@pytest.mark.parametrize("base", MODULES.values(), ids=MODULES)
def test_a_wrapper_around_the_bound_block_runs_once(calls, base, grad):
    m, x, entered = base(8).requires_grad_(False), torch.ones(1, 3, 3, 8), []
    bound = m.block

    def wrapper(*args, **kwargs):
        entered.append(1)
        return 2 * bound(*args, **kwargs)

    m.block = wrapper
    with torch.set_grad_enabled(grad):
        y = m(x)                      # forward calls the wrapper
    assert len(entered) == 1 and len(calls) == 1
    assert torch.equal(y, 2 * x)


@pytest.mark.parametrize("base", MODULES.values(), ids=MODULES)
def test_submodules_and_parameters_are_what_the_attributes_say(calls, base):
    """A property of a subclass, an attribute of the instance and a parametrised weight take precedence over the
    registered submodule or parameter of that name."""
    other = torch.nn.Linear(8, 8, bias=False)

    class Shared(base):
        @property
        def to_gate(self):
            return other

    m = Shared(8)
    m.__dict__["to_out"] = torch.nn.Linear(m.to_left.weight.shape[0], 8, bias=False)
    torch.nn.utils.parametrize.register_parametrization(m.to_left, "weight", torch.nn.Tanh())
    m.block(torch.ones(1, 3, 3, 8))
    assert calls[0]["w_gate"] is other.weight
    assert calls[0]["w_out"] is m.__dict__["to_out"].weight
    assert torch.equal(calls[0]["w_left"], m.to_left.weight) and calls[0]["w_left"] is not m.to_left.parametrizations.weight.original
    assert calls[0]["w_right"] is m.to_right.weight
