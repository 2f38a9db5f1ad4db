"""Problems whose radial matrices have another form than the generated ones:
neighbouring splines of the second radial half swapped (columns up to 8 splines
apart: the operator's slots follow the CSR order, the block-LU band is 17 wide)
and a complex overlap (the diagonal blocks' complex products).  Also the FP64
block solves with 8 warps, which mixed-precision solvers take."""
import math
import os

import numpy as np
import pytest

import oracle as O
from dirac_hydrogen_code_gb300 import formats
from dirac_hydrogen_code_gb300.cn import pulse
from dirac_hydrogen_code_gb300.gen import generate
from dirac_hydrogen_code_gb300.native import Batch, Problem, Solver

pytestmark = pytest.mark.gpu

DT = 2 * math.pi / 50.0 / 200


def _swap(path, perm):
    """Renumbers the radial basis of a block: new function i is old perm[i]."""
    m = formats.csr_read(path)
    rows = np.repeat(np.arange(m.n), np.diff(m.Ap))
    new = np.argsort(perm)
    r, c = new[rows], new[m.Ai]
    o = np.lexsort((c, r))
    m.Ap = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m.n))])
    m.Ai, m.Ax = c[o], m.Ax[o]
    formats.csr_write(path, m)


def _problem(tmp_path, ns, form):
    d = str(tmp_path)
    info = generate(dict(Nsplines=ns, Ntime=200, Nkappa=2, Nmu=0, Nl=3, rBox=30.0, Intensity=10, Omega=50.0, Cycles=1,
                         Z=1), d)
    B = 2 * (ns + 5)
    if "swapped" in form:
        perm = np.arange(B)
        k = np.arange(B // 2, B - 1, 2)
        perm[k], perm[k + 1] = k + 1, k
        for f in os.listdir(d):
            if f.endswith(".csr") and f[0] in "ghs":
                _swap(os.path.join(d, f), perm)
    if "complex" in form:
        path = os.path.join(d, "s0.csr")
        m = formats.csr_read(path)
        rows = np.repeat(np.arange(m.n), np.diff(m.Ap))
        m.Ax = m.Ax + 0.01j * np.sign(m.Ai - rows) * np.abs(m.Ax)     # stays Hermitian
        formats.csr_write(path, m)
    return Problem(d, info["lmax"]), O.load_problem(d, info["lmax"])


@pytest.mark.parametrize("form", ["swapped", "complex", "swapped complex"])
@pytest.mark.parametrize("ns", [28, 59, 93])
def test_other_layouts(tmp_path, native_lib, ns, form):
    """S x and H x of both operators within 1e-13 of |A x|'s norm of the
    oracle's matrices (a few hundred products per row), the solves with 4 and 8
    warps to a backward error of 1e-13 (65 products per row and sweep at 2^-53,
    times the condition of 32 x 32 triangles), and a step and a batch step of
    the two operators alike to the solver's tolerance."""
    prob, p = _problem(tmp_path, ns, form)
    ft = pulse(10, 50.0, 1, 70 * DT)
    S, Hst = O.stationary(p, DT)
    H = O.timedep(p, DT, ft)
    rng = np.random.default_rng(ns)
    x = rng.standard_normal(prob.n) + 1j * rng.standard_normal(prob.n)
    s = Solver(prob, DT)
    PT = (S + Hst).T.tocsr()
    for warps in (4, 8):
        s.set_precond_warps(warps)
        z = s.precond(x)
        assert np.linalg.norm(PT @ z - x) <= 1e-13 * np.linalg.norm(abs(PT) @ abs(z) + abs(x))
    bt = Batch(prob, [DT, DT])
    out = []
    for op in (0, 1):
        s.set_operator(op)
        assert s.operator()["assembled"] == op
        s.set_time(ft)
        for y, M in zip(s.apply(x, parts=True)[1:], (S, H)):
            assert np.linalg.norm(y - M @ x) <= 1e-13 * np.linalg.norm(M @ x)
        s.restart(x)
        s.step(ft, maxit=500, tol=1e-12)
        bt.set_operator(op)
        for k in range(2):
            bt.set_x(k, x)
        bt.step(np.stack([ft, ft]), maxit=500, tol=1e-12)
        out += [s.get_x(), bt.get_x(0), bt.get_x(1)]
    for y in out:
        r = (S @ x - H @ x) - (S @ y + H @ y)
        assert np.linalg.norm(r) <= 2e-12 * np.linalg.norm(S @ x - H @ x)


@pytest.mark.parametrize("form", ["", "swapped"])
def test_mixed_solver_complex128_solves(tmp_path, native_lib, form):
    """A mixed-precision solver keeps no second copy of the factors: its
    complex128 solves run in FP64 with either number of warps, to a backward
    error of 1e-13, and differ only in the order of sums."""
    prob, p = _problem(tmp_path, 60, form)
    S, Hst = O.stationary(p, DT)
    PT = (S + Hst).T.tocsr()
    rng = np.random.default_rng(5)
    b = rng.standard_normal(prob.n) + 1j * rng.standard_normal(prob.n)
    s = Solver(prob, DT, precision="mixed")
    y = []
    for warps in (4, 8):
        s.set_precond_warps(warps)
        z = s.precond(b)
        assert np.linalg.norm(PT @ z - b) <= 1e-13 * np.linalg.norm(abs(PT) @ abs(z) + abs(b))
        y.append(z)
    assert np.linalg.norm(y[0] - y[1]) <= 1e-13 * np.linalg.norm(y[0])


def test_nan_in_a_coupling_table(tmp_path, native_lib):
    """A NaN in one radial table entry reaches the same rows of the assembled
    operator as of the matrix-free one."""
    prob, p = _problem(tmp_path, 28, "")
    d, lmax = str(tmp_path), prob.info["lmax"]
    path = next(os.path.join(d, f"g{q}a{a}l{l}.csr") for l in range(lmax) for a in range(6) for q in range(4)
                if a % 2 != l % 2 and np.abs(formats.csr_read(os.path.join(d, f"g{q}a{a}l{l}.csr")).Ax).max() > 0)
    m = formats.csr_read(path)
    m.Ax[np.abs(m.Ax).argmax()] = np.nan
    formats.csr_write(path, m)
    s = Solver(Problem(d, lmax), DT)
    rng = np.random.default_rng(2)
    x = rng.standard_normal(prob.n) + 1j * rng.standard_normal(prob.n)
    fin = []
    for op in (0, 1):
        s.set_operator(op)
        s.set_time(pulse(10, 50.0, 1, 70 * DT))
        fin.append(np.isfinite(s.apply(x)))
    assert np.array_equal(fin[0], fin[1]) and not fin[0].all() and fin[0].any()
