"""Rules of the autograd layer that need no GPU, on a stand-in for the solver."""
import types

import pytest
import torch

from soliton_solver_b200 import autograd as ag

DA = 0.5


class _Quadratic:
    """E = dA/2 sum f^2; counts its gradient evaluations."""

    def __init__(self):
        self.p_f = [0, 0, 0, 0, DA]
        self.calls = 0

    def energy(self, f):
        return 0.5 * DA * float((f * f).sum())

    def energy_gradient(self, f):
        self.calls += 1
        return f.clone()

    def energy_vjp(self, f, g):
        self.calls += 1
        return f * (g.to(f.dtype) * DA)

    def observables(self, f, names):
        return {n: 0.0 for n in names}


def test_batched_backward_evaluates_the_gradient_once():
    s = _Quadratic()
    x = torch.randn(5, dtype=torch.float64, requires_grad=True)
    w = torch.tensor([1.0, -2.0, 3.0], dtype=torch.float64)
    (g,) = torch.autograd.grad(ag.energy(x, s), x, grad_outputs=w, is_grads_batched=True)
    torch.testing.assert_close(g, DA * w[:, None] * x.detach(), rtol=1e-15, atol=0)
    assert s.calls == 1


@pytest.mark.parametrize("theory", ["baby_skyrme", "ginzburg_landau_superconductor"])
@pytest.mark.parametrize("name", ["energy", "skyrmion", "vortex", "nonsense"])
def test_only_couplings_have_coupling_gradients(theory, name):
    sim = types.SimpleNamespace(theory=types.SimpleNamespace(__name__=f"theories.{theory}"), solver=_Quadratic(),
                                Field=torch.zeros(3))
    with pytest.raises(KeyError):
        ag.coupling_gradients(sim, ("kappa", name))
    assert ag.coupling_gradients(sim, ()) == {}
