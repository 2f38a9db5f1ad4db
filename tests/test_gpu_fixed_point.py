"""The assembled operator (fixed-point products) against the matrix-free one
(FP64) of the same solver, at block sizes on the edges of the row chunks:
full chunks, one spline more or less, odd halves, a single short chunk; and
the preconditioner's fixed-point solves at the edges of their chunks."""
import math

import numpy as np
import pytest

import oracle as O
from dirac_hydrogen_code_gb300.cn import pulse
from dirac_hydrogen_code_gb300.gen import generate
from dirac_hydrogen_code_gb300.native import Problem, Solver

pytestmark = pytest.mark.gpu

# NSplines + 5 splines per half: 22, 32, 33, 63, 64, 65, 129
SIZES = [17, 27, 28, 58, 59, 60, 124]


def _problem(tmp_path, ns, nkappa=2, nmu=0, nl=3):
    p = dict(Nsplines=ns, Ntime=60, Nkappa=nkappa, Nmu=nmu, Nl=nl, rBox=30.0, Intensity=10, Omega=50.0, Cycles=1, Z=1)
    info = generate(p, str(tmp_path))
    prob = Problem(str(tmp_path), info["lmax"])
    dt = 2 * math.pi / 50.0 / 60
    return prob, dt, pulse(10, 50.0, 1, 20 * dt)


@pytest.mark.parametrize("ns", SIZES)
def test_assembled_matches_matrix_free(tmp_path, native_lib, ns):
    """S x and H x within 2e-14 of |A x|'s norm (FP64 sums of ~100 products
    round to ~1e-15, the fixed-point ones to less), for entries spread over
    24 orders of magnitude, and the same non-finite rows for a NaN and an
    infinity in one entry of x."""
    prob, dt, ft = _problem(tmp_path, ns)
    rng = np.random.default_rng(ns)
    x = (rng.standard_normal(prob.n) + 1j * rng.standard_normal(prob.n)) * 10.0 ** rng.uniform(-24, 0, prob.n)
    s = Solver(prob, dt)
    out = {}
    for op in (0, 1):
        s.set_operator(op)
        s.set_time(ft)
        out[op] = s.apply(x, parts=True)
    for a, b in zip(out[0], out[1]):
        assert np.linalg.norm(a - b) <= 2e-14 * np.linalg.norm(a)
    for bad in (complex(np.nan, 0.0), complex(1.0, np.inf)):
        xb = x.copy()
        xb[int(rng.integers(prob.n))] = bad
        fin = []
        for op in (0, 1):
            s.set_operator(op)
            s.set_time(ft)
            fin.append(np.isfinite(s.apply(xb)))
        assert np.array_equal(fin[0], fin[1]) and not fin[0].all()


def test_zero_field_and_tiny_state(tmp_path, native_lib):
    """f(t) = 0 leaves S + i h dt/2 h0; a state at 1e-280 keeps its product
    to rounding."""
    prob, dt, ft = _problem(tmp_path, 28)
    rng = np.random.default_rng(3)
    x = rng.standard_normal(prob.n) + 1j * rng.standard_normal(prob.n)
    s = Solver(prob, dt)
    for f, scale in ((np.zeros(6, complex), 1.0), (ft, 1e-280)):
        y = []
        for op in (0, 1):
            s.set_operator(op)
            s.set_time(f)
            y.append(s.apply(scale * x) / scale)
        assert np.linalg.norm(y[0] - y[1]) <= 2e-14 * np.linalg.norm(y[0])


# rows per block 30, 32, 34, 64, 66, 96, 128, 130, 256, 258: one chunk of 32
# (full, ragged), odd and even chunk counts, a ragged last chunk
PRECOND_SIZES = [10, 11, 12, 27, 28, 43, 59, 60, 123, 124]


@pytest.mark.parametrize("ns", PRECOND_SIZES)
def test_preconditioner_chunks(tmp_path, native_lib, ns):
    """Normwise backward error of every block row's solve within 1e-13 (49
    products per row and sweep at 2^-53, times the condition of 32 x 32
    triangles, some 20), for entries of one size, spread over 24 orders of
    magnitude, tiny, and zero but for one chunk; a NaN in one block row makes
    that row's result NaN and leaves the others' bits."""
    prob, dt, _ = _problem(tmp_path, ns)
    p = O.load_problem(str(tmp_path), prob.info["lmax"])
    S, Hst = O.stationary(p, dt)
    PT = (S + Hst).T.tocsr()
    B = 2 * (ns + 5)
    nblk = prob.n // B
    rng = np.random.default_rng(ns)
    x = rng.standard_normal(prob.n) + 1j * rng.standard_normal(prob.n)
    one = np.zeros_like(x)
    at = int(rng.integers(B))
    one.reshape(nblk, B)[:, at] = x.reshape(nblk, B)[:, at]
    s = Solver(prob, dt)

    def rows(v):
        return np.linalg.norm(v.reshape(nblk, B), axis=1)

    y = {}
    for name, b in (("even", x), ("spread", x * 10.0 ** rng.uniform(-24, 0, prob.n)), ("tiny", 1e-280 * x), ("one", one)):
        y[name] = s.precond(b)
        k = 1e280 if name == "tiny" else 1.0
        z, b = k * y[name], k * b
        assert (rows(PT @ z - b) <= 1e-13 * rows(abs(PT) @ abs(z) + abs(b))).all(), name
    xb = x.copy()
    xb[B + at] = np.nan
    yb = s.precond(xb).reshape(nblk, B)
    assert np.isnan(yb[1]).all()
    keep = np.arange(nblk) != 1
    assert np.array_equal(yb[keep], y["even"].reshape(nblk, B)[keep])
