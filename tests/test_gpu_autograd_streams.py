"""The autograd ops called on another stream than the solver's: a grad_E that is written late on the
caller's stream, and a solver's stream that is busy, give the same gradient as everything on one
stream (scaled by another kernel: two roundings of 6e-8)."""
import pytest
import torch

from soliton_solver_b200.autograd import energy
from soliton_solver_b200.core.solver import Solver
from soliton_solver_b200.theories import load_theory

pytestmark = pytest.mark.gpu

BUSY = 100_000_000  # clock cycles, about 50 ms


def _solver(stream):
    theory = load_theory("Abelian Higgs")
    rp = theory.params.default_params(xlen=96, ylen=128, lsx=0.1, lsy=0.1).resolved()
    p_i, p_f = theory.params.pack_device_params(rp)
    s = Solver(theory.kernels.THEORY_ID, p_i, p_f, "fp32", stream=stream)
    g = torch.Generator(device="cuda").manual_seed(1)
    f = 0.5 + 0.1 * torch.randn(int(rp.dim_fields), device="cuda", generator=g)
    s.bind(f, torch.zeros_like(f))
    return s, f


@pytest.mark.parametrize("bound", ["default", "own"])
@pytest.mark.parametrize("busy", ["caller", "solver"])
def test_backward_on_another_stream(bound, busy):
    own = torch.cuda.Stream()
    s, f = _solver(None if bound == "default" else own)
    want = s.energy_gradient(f) * (2.5 * float(s.p_f[4]))
    torch.cuda.synchronize()
    solver_stream = torch.cuda.default_stream() if bound == "default" else own
    side = torch.cuda.Stream()
    leaf = f.clone().requires_grad_(True)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        E = energy(leaf, s)
        grad_E = torch.zeros((), dtype=torch.float64, device="cuda")
        with torch.cuda.stream(side if busy == "caller" else solver_stream):
            torch.cuda._sleep(BUSY)
        grad_E.fill_(2.5)
        E.backward(grad_E)
        got = leaf.grad.clone()
    torch.cuda.synchronize()
    torch.testing.assert_close(got, want, rtol=2e-7, atol=0)
