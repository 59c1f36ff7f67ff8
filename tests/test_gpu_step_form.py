"""Which form of the step a lattice takes, and the plain-row two-launch step at odd counts.

Tiles of 8 x 32, 16 x 32 and 16 x 64 sites run cooperatively while all are resident.  For FP32 and four
components shared memory and registers allow 3, 3 and 2 CTAs per SM (444, 444 and 296 tiles on 148 SMs):
420 x 500 makes 848 and 432 tiles, 500 x 480 makes 945, 480 and 256; six components take 2 CTAs of the
first.  No tile shape holds 10^6 sites."""
import math

import numpy as np
import pytest
import torch

from soliton_solver_b200.core.solver import Solver
from soliton_solver_b200.theories import load_theory

pytestmark = pytest.mark.gpu

KW = {"Chiral magnet": dict(dmi_term="Heusler", demag=True, B=0.2, unit_magnetization=True, lsx=0.05, lsy=0.05),
      "Baby Skyrme": dict(unit_magnetization=True, lsx=0.1, lsy=0.1, time_step=0.02),
      "Abelian Higgs": dict(lsx=0.1, lsy=0.1),
      "s+id superconductor": dict(lsx=0.1, lsy=0.1)}


def _solver(th, prec, X, Y):
    theory = load_theory(th)
    rp = theory.params.default_params(xlen=X, ylen=Y, **KW[th]).resolved()
    p_i, p_f = theory.params.pack_device_params(rp)
    rng = np.random.default_rng(X + Y)
    F = np.zeros((rp.number_total_fields, X, Y))
    for a, v in enumerate(theory.initial_config.vacuum(rp)):
        F[a] = v
    F += 0.05 * rng.standard_normal(F.shape)
    if "unit_magnetization" in KW[th]:
        F[:3] /= np.sqrt((F[:3] ** 2).sum(0))
    s = Solver(theory.kernels.THEORY_ID, p_i, p_f, prec)
    f = torch.tensor(F.reshape(-1), dtype=s.dtype, device="cuda")
    s.bind(f, torch.zeros_like(f))
    return s


@pytest.mark.parametrize("th,prec,X,Y,form", [
    *[(th, prec, 64, 100, 1) for th in sorted(KW) for prec in ("fp32", "fp64")],
    *[(th, prec, 1000, 1000, 0) for th in sorted(KW) for prec in ("fp32", "fp64")],
    ("Chiral magnet", "fp32", 420, 500, 2), ("Chiral magnet", "fp32", 500, 480, 3),
    ("Abelian Higgs", "fp32", 420, 500, 2), ("Abelian Higgs", "fp32", 500, 480, 3),
    ("s+id superconductor", "fp32", 200, 203, 1)])
def test_form(th, prec, X, Y, form):
    s = _solver(th, prec, X, Y)
    assert s.step_form == form
    s.set_variant(6, 1)
    assert s.step_form == 0
    assert Solver(s.theory_id, s.p_i, s.p_f, "plain_fp64").step_form == 0


@pytest.mark.parametrize("th", sorted(KW))
@pytest.mark.parametrize("prev", [1e300, -1e300], ids=["free", "arrested"])
def test_odd_counts_of_the_plain_two_launch_step(th, prev):
    """One call of seven steps and its splits into odd and even ones, where an odd call copies the field and
    the velocity back: the same kernels on the same values, bitwise."""
    outs = []
    for split in ([7], [1, 2, 1, 3], [3, 3, 1]):
        s = _solver(th, "fp32", 256, 150 if th != "Baby Skyrme" else 151)
        s.set_variant(6, 1)
        assert s.step_form == 0 and not s.tma_enabled
        Es = [s.step(k, prev if i == 0 else math.nan)[0] for i, k in enumerate(split)]
        outs.append((np.concatenate(Es), s.field.cpu().numpy(), s.velocity.cpu().numpy()))
    for got in outs[1:]:
        for a, b in zip(got, outs[0]):
            np.testing.assert_array_equal(a, b)


def test_fp64_second_phase_variants():
    """Phase B has both variants in FP64 too: pinned to one tile per CTA and back, the same step up to the
    compiler's contraction in the two kernels (1e-12 of max|phi|); a handle pinned to neither has variant 1."""
    outs = []
    for pins in ((), (0,), (0, 1)):
        s = _solver("Abelian Higgs", "fp64", 600, 640)
        assert s.step_form == 0 and s._lib.ss_get_variant(s._h, 4) == 1
        for v in pins:
            s.set_variant(4, v)
            assert s._lib.ss_get_variant(s._h, 4) == v
        s.step(5, 1e300)
        outs.append(s.field)
    assert torch.equal(outs[0], outs[2])
    assert (outs[0] - outs[1]).abs().max() <= 1e-12 * outs[0].abs().max()


def test_refused_variant_leaves_the_step_form():
    s = _solver("Chiral magnet", "fp32", 64, 101)
    assert s.step_form == 1 and not s.tma_enabled
    with pytest.raises(Exception, match="TMA"):
        s.set_variant(4, 1)
    assert s.step_form == 1
    s = _solver("Chiral magnet", "fp64", 64, 100)
    with pytest.raises(ValueError, match="no pipelined variant"):
        s.set_variant(1, 1)
    assert s.step_form == 1
