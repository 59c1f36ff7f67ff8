"""Field, velocity and output buffers aligned to their element type only (views that start one
element into their storage): the interior tiles' two-site accesses fall back to single ones.
Against the same call on aligned buffers.  Rows of even length that are no multiple of 16 bytes
(FP32) are staged by plain loads either way and give the same bits; FP64 rows of even length are
staged by TMA when aligned, which rounds T2 and T3 differently (one rounding of 1.1e-16 each),
and the compiler may contract differently: 1e-12 of max|phi| over five steps, as between the
cooperative and the two-launch step."""
import ctypes

import numpy as np
import pytest
import torch

from soliton_solver_b200 import _native as nat
from soliton_solver_b200.core.batch import BatchSolver
from soliton_solver_b200.core.solver import Solver
from soliton_solver_b200.theories import load_theory

pytestmark = pytest.mark.gpu

KW = {"Chiral magnet": dict(dmi_term="Heusler", demag=True, B=0.2, unit_magnetization=True, lsx=0.05, lsy=0.05),
      "s+id superconductor": dict(lsx=0.1, lsy=0.1)}


def _off(t):
    """A copy of t one element into its storage."""
    s = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    s[1:] = t
    return s[1:]


def _case(th, X, Y, prec):
    theory = load_theory(th)
    rp = theory.params.default_params(xlen=X, ylen=Y, **KW[th]).resolved()
    rng = np.random.default_rng(X + Y)
    F = np.zeros((rp.number_total_fields, X, Y))
    for a, v in enumerate(theory.initial_config.vacuum(rp)):
        F[a] = v
    F += 0.05 * rng.standard_normal(F.shape)
    if "unit_magnetization" in KW[th]:
        F[:3] /= np.sqrt((F[:3] ** 2).sum(0))
    V = 0.05 * rng.standard_normal(F.shape)
    dt = torch.float32 if prec == "fp32" else torch.float64
    f, v = (torch.tensor(a.reshape(-1), dtype=dt, device="cuda") for a in (F, V))
    return theory, rp, f, v


def _close(got, want, prec, scale=None):
    if prec == "fp32":
        assert torch.equal(got, want)
    else:
        assert (got - want).abs().max() <= 1e-12 * max(float(want.abs().max()), float(scale or 0.0))


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("th", sorted(KW))
@pytest.mark.parametrize("X,Y,pinned", [(120, 150, False), (120, 150, True), (40, 70, True), (700, 630, False)])
def test_step(th, prec, X, Y, pinned):
    theory, rp, f0, v0 = _case(th, X, Y, prec)
    p_i, p_f = theory.params.pack_device_params(rp)
    outs = []
    for view in (torch.clone, _off):
        s = Solver(theory.kernels.THEORY_ID, p_i, p_f, prec)
        f, v = view(f0), view(v0)
        s.bind(f, v)
        if pinned:
            s.set_variant(6, 1)
        E1, _ = s.step(3, 1e300)
        E2, _ = s.step(2)
        outs.append((f, v, np.concatenate([E1, E2]), s.energy(f)))
    (fa, va, Ea, ea), (fb, vb, Eb, eb) = outs
    _close(fb, fa, prec)
    _close(vb, va, prec, fa.abs().max())
    np.testing.assert_allclose(Eb, Ea, rtol=1e-12, atol=1e-12 * X * Y)
    np.testing.assert_allclose(eb, ea, rtol=1e-12, atol=1e-12 * X * Y)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("th", sorted(KW))
@pytest.mark.parametrize("Y", [150, 192])
def test_gradient_outputs(th, prec, Y):
    theory, rp, f, v = _case(th, 120, Y, prec)
    p_i, p_f = theory.params.pack_device_params(rp)
    s = Solver(theory.kernels.THEORY_ID, p_i, p_f, prec)
    s.bind(f, v)
    outs = []
    for view in (torch.clone, _off):
        eg, l, g, w = (view(torch.zeros_like(f)) for _ in range(4))
        s.gradient(f, eg, l)
        s.energy_gradient(f, g)
        s.energy_vjp(f, torch.full((), 2.5, dtype=torch.float64, device="cuda"), w)
        outs.append((eg, l, g, w))
    for a, b in zip(*outs):
        _close(b, a, prec)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_batch(prec):
    theory, rp, f0, v0 = _case("Chiral magnet", 100, 150, prec)
    outs = []
    for view in (torch.clone, _off):
        b = BatchSolver(theory, [rp, rp], prec)
        b.fields = [view(f0), view(f0)]
        b.velocities = [view(v0), view(v0)]
        ptrs = [(ctypes.c_void_p * 2)(*(t.data_ptr() for t in ts)) for ts in (b.fields, b.velocities)]
        nat.check(b._lib.ss_batch_bind(b._h, *ptrs, b.workspace.data_ptr(), b.workspace.numel(),
                                       torch.cuda.current_stream().cuda_stream))
        b.step(5, 1e300)
        outs.append((b.fields[1], b.velocities[1]))
    (fa, va), (fb, vb) = outs
    _close(fb, fa, prec)
    _close(vb, va, prec, fa.abs().max())
