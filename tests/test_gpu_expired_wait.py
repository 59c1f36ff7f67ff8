"""An expired wait of the cooperative step (its grid barrier) is reported, by every call until the
status has been read, and leaves nothing behind: the next step, without a re-bind, is the step of
a fresh handle.  The hook makes the barrier expect one CTA more than there are.  The lattice has
rows that are no multiple of 16 bytes, so the two-launch step would wait for nothing and a timeout
shows that the cooperative step ran."""
import numpy as np
import pytest
import torch

from soliton_solver_b200._native import DeviceTimeoutError
from soliton_solver_b200.core.solver import Solver
from soliton_solver_b200.theories import load_theory

pytestmark = pytest.mark.gpu

WAIT = 2_000_000_000


def _solver(X=200, Y=151):
    theory = load_theory("Chiral magnet")
    rp = theory.params.default_params(xlen=X, ylen=Y, lsx=0.05, lsy=0.05, dmi_term="Heusler", demag=True,
                                      unit_magnetization=True).resolved()
    p_i, p_f = theory.params.pack_device_params(rp)
    m = np.random.default_rng(1).standard_normal((3, X, Y)) * 0.1
    m[2] += 1.0
    F = np.concatenate([m / np.sqrt((m * m).sum(0)), np.zeros((1, X, Y))]).reshape(-1)
    s = Solver(theory.kernels.THEORY_ID, p_i, p_f, "fp32")
    f = torch.tensor(F, dtype=torch.float32, device="cuda")
    start = f.clone()
    s.bind(f, torch.zeros_like(f))
    assert not s.tma_enabled
    return s, start


def _step(s, start, n=3):
    s.field.copy_(start)
    s.velocity.zero_()
    E, err = s.step(n, 1e300)
    return E, err, s.field.cpu().numpy(), s.velocity.cpu().numpy()


def test_expired_grid_barrier_is_reported_and_leaves_nothing_behind():
    want = _step(*_solver())
    s, start = _solver()
    for _ in range(2):
        s.debug_wait_timeout(200_000, inject=True)  # 3.2e6 cycles: under 2 ms
        with pytest.raises(DeviceTimeoutError):
            s.step(3, 1e300)
        s.debug_wait_timeout(WAIT, inject=False)
        for a, b in zip(_step(s, start), want):
            np.testing.assert_array_equal(a, b)


def test_launches_behind_an_expired_barrier_fail_until_it_is_reported():
    s, start = _solver()
    want = _step(s, start)
    s.debug_wait_timeout(200_000, inject=True)  # 3.2e6 cycles: under 2 ms
    s.step_async(3, 1e300)
    s.debug_wait_timeout(WAIT, inject=False)
    E = torch.full((3,), 7.0, dtype=torch.float64, device="cuda")
    s.step_async(3, 1e300, E)
    with pytest.raises(DeviceTimeoutError):
        s.check_status()
    assert (E == 7.0).all()  # no energy of a step that did not run
    s.check_status()
    for a, b in zip(_step(s, start), want):
        np.testing.assert_array_equal(a, b)


def test_longest_wait_does_not_overflow():
    s, start = _solver()
    want = _step(s, start)
    s.debug_wait_timeout(2**63 - 1, inject=False)
    for a, b in zip(_step(s, start), want):
        np.testing.assert_array_equal(a, b)
