"""Several totals in one pass against the single calls, and the energy's one-pass backward
against its composition, on tiles' edges, remainders and rows that are no multiple of 16 bytes.

The one-pass totals take the same jets in the same order per site and the same tiles as the
single ones: equal bitwise for FP32 fields and for charges and couplings (FP64 energies are the
flow's own in both).  The backward multiplies each row once by the same rounded factor: bitwise."""
import numpy as np
import pytest
import torch

from soliton_solver_b200.autograd import energy
from soliton_solver_b200.core.solver import Solver
from soliton_solver_b200.theories import load_theory

pytestmark = pytest.mark.gpu

CASES = {"Chiral magnet": (dict(dmi_term="Heusler", demag=True, B=0.2, unit_magnetization=True, lsx=0.05, lsy=0.05),
                           ["energy", "skyrmion", "magnetic", "coup_K", "coup_h", "coup_mu"]),
         "Baby Skyrme": (dict(unit_magnetization=True, lsx=0.1, lsy=0.1), ["energy", "skyrmion", "kappa", "mpi"]),
         "Abelian Higgs": (dict(lsx=0.1, lsy=0.1), ["energy", "vortex", "Lambda"]),
         "s+id superconductor": (dict(lsx=0.1, lsy=0.1), ["energy", "vortex"])}


def _solver(th, prec, X, Y):
    theory = load_theory(th)
    rp = theory.params.default_params(xlen=X, ylen=Y, **CASES[th][0]).resolved()
    p_i, p_f = theory.params.pack_device_params(rp)
    F = np.zeros((rp.number_total_fields, X, Y))
    for a, v in enumerate(theory.initial_config.vacuum(rp)):
        F[a] = v
    F += 0.1 * np.random.default_rng(X + Y).standard_normal(F.shape)
    s = Solver(theory.kernels.THEORY_ID, p_i, p_f, prec)
    f = torch.tensor(F.reshape(-1), dtype=torch.float32 if prec == "fp32" else torch.float64, device="cuda")
    s.bind(f, torch.zeros_like(f))
    return s, f


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("th", sorted(CASES))
@pytest.mark.parametrize("X,Y", [(1, 1), (16, 64), (17, 65), (100, 203), (129, 320)])
def test_totals_in_one_pass_equal_the_single_ones(th, prec, X, Y):
    s, f = _solver(th, prec, X, Y)
    names = CASES[th][1]
    got = s.observables(f, names)
    for n in names:
        want = s.energy(f) if n == "energy" else s.charge(f, n) if n in ("skyrmion", "magnetic", "vortex") else \
            s.coupling_grad(f, n)
        assert got[n] == want, n


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("th", sorted(CASES))
@pytest.mark.parametrize("X,Y", [(17, 65), (128, 320)])
def test_backward_in_one_pass_equals_its_composition(th, prec, X, Y):
    s, f = _solver(th, prec, X, Y)
    leaf = f.clone().requires_grad_(True)
    (3.7 * energy(leaf, s)).backward()
    factor = torch.full((), 3.7, dtype=torch.float64, device="cuda").to(f.dtype) * float(s.p_f[4])
    torch.testing.assert_close(leaf.grad, s.energy_gradient(f) * factor, rtol=0, atol=0)
