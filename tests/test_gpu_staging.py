"""Handles that come and go, in several threads, share a few page-locked staging blocks: each call's
trajectory and energy are its own (bitwise those of the same calls alone)."""
import threading

import numpy as np
import pytest
import torch

from soliton_solver_b200.core.solver import Solver
from soliton_solver_b200.theories import load_theory

pytestmark = pytest.mark.gpu


def _run(seed, X, Y):
    theory = load_theory("Abelian Higgs")
    p_i, p_f = theory.params.pack_device_params(theory.params.default_params(xlen=X, ylen=Y, lsx=0.1, lsy=0.1).resolved())
    s = Solver(theory.kernels.THEORY_ID, p_i, p_f, "fp32")
    rng = np.random.default_rng(seed)
    f = torch.tensor(0.5 + 0.05 * rng.standard_normal(s.nf * s.N), dtype=torch.float32, device="cuda")
    s.bind(f, torch.zeros_like(f))
    E0 = s.energy(f)
    E, err = s.step(5, 1e300)
    return np.concatenate([[E0], E, err, [s.energy(f)]])


def test_short_lived_handles_in_threads():
    jobs = [(i, 40 + 8 * i, 64 if i % 2 else 600) for i in range(7)]
    want = [_run(*j) for j in jobs]
    got = [[] for _ in jobs]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(8):
                got[i].append(_run(*jobs[i]))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join(timeout=120)
    for g, w in zip(got, want):
        assert len(g) == 8
        for r in g:
            np.testing.assert_array_equal(r, w)
