"""The residual |b - A x| / |b| of a solved step, formed from the oracle's
matrices: the solver's own is a recurrence, and what its products leave out
does not show there."""
import math

import numpy as np
import pytest

import oracle as O
from dirac_hydrogen_code_gb300.cn import pulse
from dirac_hydrogen_code_gb300.gen import generate
from dirac_hydrogen_code_gb300.native import Batch, Problem, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [27, 124])
def test_true_residual_of_a_step(tmp_path, native_lib, ns):
    """From a random state (the first residual is as large as b) at the
    default tolerance: the assembled operator leaves no more than the
    matrix-free one, whose products round more often; 1.25 covers the scatter
    of two rms values over some 800 and 3,100 rows.  One pulse and a batch."""
    ntime = 60
    p = dict(Nsplines=ns, Ntime=ntime, Nkappa=2, Nmu=0, Nl=3, rBox=30.0, Intensity=10, Omega=50.0, Cycles=1, Z=1)
    info = generate(p, str(tmp_path))
    prob, p = Problem(str(tmp_path), info["lmax"]), O.load_problem(str(tmp_path), info["lmax"])
    dt = 2 * math.pi / 50.0 / ntime
    ft = pulse(10, 50.0, 1, 20 * dt)
    S, _ = O.stationary(p, dt)
    H = O.timedep(p, dt, ft)
    rng = np.random.default_rng(ns)
    x = rng.standard_normal(prob.n) + 1j * rng.standard_normal(prob.n)
    b = S @ x - H @ x

    def residual(y):
        return np.linalg.norm(b - S @ y - H @ y) / np.linalg.norm(b)

    s, bt = Solver(prob, dt), Batch(prob, [dt, dt])
    res = []
    for op in (0, 1):
        s.set_operator(op)
        s.restart(x)
        s.step(ft, maxit=500)
        bt.set_operator(op)
        for k in range(2):
            bt.set_x(k, x)
        bt.step(np.stack([ft, ft]), maxit=500)
        res.append([residual(s.get_x()), residual(bt.get_x(0)), residual(bt.get_x(1))])
    assert all(a <= 1.25 * m for m, a in zip(*res)), res
