"""The cooperative step (small lattices, all steps of a call in one launch) against the step
as two launches (a pinned handle) from the same state: sizes at the edges of its tiles
(8 x 32, 16 x 32 and 16 x 64 sites), remainders, rows that are no multiple of 16 bytes, the
smallest lattices and the largest of each shape, odd and even step counts, arrests.

Both run the same per-site arithmetic.  FP32: packed operations with explicit rounding in the
same order, so the fields agree bitwise; energies are FP64 sums of the same site values over
other tiles: 1e-12.  FP64: the compiler may contract a * b + c differently in the two kernels,
one rounding (1.1e-16) per operation; a step is stable (dt times the highest frequency is
below RK4's 2.8) and sums ~100 operations per site, so 1e-12 of max|phi| for the field and the
energy over 5 steps."""
import math
import threading

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


def _case(th, X, Y, seed):
    theory = load_theory(th)
    rp = theory.params.default_params(xlen=X, ylen=Y, **KW[th]).resolved()
    p_i, p_f = theory.params.pack_device_params(rp)
    rng = np.random.default_rng(seed)
    F = np.zeros((rp.number_total_fields, X, Y))
    for a, v in enumerate(theory.initial_config.vacuum(rp)):
        F[a] = v
    F += 0.05 * rng.standard_normal(F.shape)
    if "unit_magnetization" in KW[th]:
        F[:3] /= np.sqrt((F[:3] ** 2).sum(0))
    V = 0.05 * rng.standard_normal(F.shape)
    return theory.kernels.THEORY_ID, p_i, p_f, F.reshape(-1), V.reshape(-1)


def _run(case, prec, split, prev, pinned):
    tid, p_i, p_f, F, V = case
    dt = torch.float32 if prec == "fp32" else torch.float64
    s = Solver(tid, p_i, p_f, prec)
    f = torch.tensor(F, dtype=dt, device="cuda")
    v = torch.tensor(V, dtype=dt, device="cuda")
    s.bind(f, v)
    if pinned:
        s.set_variant(6, 1)
    Es, errs = [], []
    for i, k in enumerate(split):
        E, err = s.step(k, prev if i == 0 else math.nan)
        Es.extend(E)
        errs.extend(err)
    return np.array(Es), np.array(errs), f.cpu().numpy(), v.cpu().numpy()


SIZES = [(1, 1), (3, 5), (8, 32), (9, 33), (7, 31), (64, 100), (65, 130), (201, 203), (320, 336), (420, 500), (500, 600),
         (530, 560)]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("th", sorted(KW))
@pytest.mark.parametrize("X,Y", SIZES, ids=[f"{x}x{y}" for x, y in SIZES])
def test_cooperative_step_equals_two_launches(th, prec, X, Y):
    case = _case(th, X, Y, 3)
    # the first test arrests (every energy is above -1e300), the following ones as the flow has it
    want = _run(case, prec, [5], -1e300, True)
    for split in ([5], [2, 3]):
        got = _run(case, prec, split, -1e300, False)
        if prec == "fp32":
            np.testing.assert_array_equal(got[2], want[2])
            np.testing.assert_array_equal(got[3], want[3])
            np.testing.assert_array_equal(got[1], want[1])
        else:
            scale = np.abs(want[2]).max()
            assert np.abs(got[2] - want[2]).max() <= 1e-12 * scale
            assert np.abs(got[3] - want[3]).max() <= 1e-12 * max(np.abs(want[3]).max(), scale)
            np.testing.assert_allclose(got[1], want[1], rtol=1e-10)
        np.testing.assert_allclose(got[0], want[0], rtol=1e-12, atol=1e-12 * X * Y)


def test_cooperative_steps_on_concurrent_streams():
    """Two threads step their own lattices on their own streams; each result is that of the
    same steps alone."""
    cases = [_case("Chiral magnet", 256, 256, 1), _case("Baby Skyrme", 200, 256, 2)]
    want = [_run(c, "fp32", [200], 1e300, False) for c in cases]
    got = [None, None]

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            got[i] = _run(cases[i], "fp32", [40] * 5, 1e300, False)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(timeout=120)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g[2], w[2])
        np.testing.assert_array_equal(g[0], w[0])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("Y", [192, 150], ids=["tma", "plain"])
def test_mispredicted_arrest(prec, Y):
    """Saddle flow as two launches: two arrested steps make the next step's first kernel leave
    l2 out; the energy of the smooth field falls instead, so l2 comes from the extra kernel.
    Against one-step calls, which never predict.  FP32 bitwise; FP64 as above."""
    case = _case("Chiral magnet", 256, Y, 5)
    tid, p_i, p_f, F, V = case
    dt = torch.float32 if prec == "fp32" else torch.float64
    # a long-wave texture at rest with a weak demag coupling runs downhill for many steps
    p_f = p_f.copy()
    p_f[8] = 1e-3
    x, y = np.meshgrid(np.arange(256), np.arange(Y), indexing="ij")
    m = np.stack([0.4 * np.sin(0.2 * x), 0.4 * np.cos(0.15 * y), np.ones_like(x, dtype=float)])
    F = np.concatenate([m / np.sqrt((m * m).sum(0)), np.zeros((1, 256, Y))]).reshape(-1)
    V = np.zeros_like(V)
    outs = []
    for split in ([5], [1] * 5):
        s = Solver(tid, p_i, p_f, prec)
        f, v = (torch.tensor(a, dtype=dt, device="cuda") for a in (F, V))
        s.bind(f, v)
        s.set_variant(6, 1)
        for _ in range(3):
            s.step(1, -1e300)
        f.copy_(torch.tensor(F, dtype=dt))
        v.copy_(torch.tensor(V, dtype=dt))
        Es = []
        for i, k in enumerate(split):
            Es.extend(s.step(k, 1e300 if i == 0 else math.nan)[0])
        assert Es[0] < 1e300 and Es[1] < Es[0]  # the prediction was wrong
        outs.append((np.array(Es), f.cpu().numpy(), v.cpu().numpy()))
    (Ea, fa, va), (Eb, fb, vb) = outs
    if prec == "fp32":
        np.testing.assert_array_equal(fa, fb)
        np.testing.assert_array_equal(va, vb)
    else:
        assert np.abs(fa - fb).max() <= 1e-12 * np.abs(fb).max()
        assert np.abs(va - vb).max() <= 1e-12 * max(np.abs(vb).max(), np.abs(fb).max())
    np.testing.assert_allclose(Ea, Eb, rtol=1e-12)
