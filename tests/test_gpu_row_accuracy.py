"""Accuracy of single rows.  The fixed-point products must leave every row of
a result as accurate as FP64 products do: the error of a row is measured
against the sum of the magnitudes of that row's own terms, for vectors whose
entries span many orders of magnitude within a block row (radial functions
that start as a power of r, decaying tails, random spreads)."""
import copy
import math

import numpy as np
import pytest

import oracle as O
from dirac_hydrogen_code_gb300.cn import pulse
from dirac_hydrogen_code_gb300.gen import generate
from dirac_hydrogen_code_gb300.native import Problem, Solver

pytestmark = pytest.mark.gpu

OMEGA, NTIME = 50.0, 60
DT = 2 * math.pi / OMEGA / NTIME


def _problem(tmp_path, ns, nkappa=2):
    p = dict(Nsplines=ns, Ntime=NTIME, Nkappa=nkappa, Nmu=0, Nl=3, rBox=30.0, Intensity=10, Omega=OMEGA, Cycles=1, Z=1)
    info = generate(p, str(tmp_path))
    return Problem(str(tmp_path), info["lmax"]), O.load_problem(str(tmp_path), info["lmax"])


def _vectors(nblk, B, rng):
    """Block vectors by name: r^p starts, growth and decay over 24 orders of
    magnitude along the radius, and a random spread of entries."""
    t = np.tile(np.linspace(0.0, 1.0, B // 2), 2)
    ph = np.exp(2j * math.pi * rng.uniform(size=(nblk, 1)))
    z = rng.standard_normal((nblk, B)) + 1j * rng.standard_normal((nblk, B))
    out = {"r^%d" % p: ph * (t + 1e-3) ** p * np.exp(-8 * t) for p in (1, 3, 5, 7)}
    out["grow"], out["decay"] = z * 10.0 ** (24 * (t - 1)), z * 10.0 ** (-24 * t)
    out["spread"] = z * 10.0 ** rng.uniform(-24, 0, (nblk, B))
    return {k: np.ascontiguousarray(v.reshape(-1)) for k, v in out.items()}


@pytest.mark.parametrize("ns", [27, 60, 124, 250])
def test_operator_rows(tmp_path, native_lib, ns):
    """S x and H x of the assembled operator, each row within 1e-14 of the
    sum of its terms' magnitudes (angular x radial x field x vector): a few
    hundred products and as many roundings of the values, whose random walk
    is ~25 x 2^-53 on each side.  The matrix-free operator meets the same
    bound."""
    prob, p = _problem(tmp_path, ns)
    ft = pulse(10, OMEGA, 1, 20 * DT)
    S, _ = O.stationary(p, DT)
    H = O.timedep(p, DT, ft)
    pa = copy.copy(p)
    for name in ("H0", "H1", "g", "gt", "h0", "s0", "kappa"):
        v = getattr(p, name)
        setattr(pa, name, [abs(a) for a in v] if isinstance(v, list) else abs(v))
    Sa, Ha = abs(O.stationary(pa, DT)[0]), abs(O.timedep(pa, DT, abs(ft)))
    B = 2 * (ns + 5)
    s = Solver(prob, DT)
    for name, x in _vectors(prob.n // B, B, np.random.default_rng(ns)).items():
        for op in (0, 1):
            s.set_operator(op)
            s.set_time(ft)
            for y, M, A in zip(s.apply(x, parts=True)[1:], (S, H), (Sa, Ha)):
                err, mag = np.abs(y - M @ x), A @ np.abs(x)
                assert (err <= 1e-14 * mag).all(), (name, op, float((err / mag).max()))


def _factors(A):
    """Block-LU sweeps' factors of A (in the factors' order): inverse triangles
    and the 16 chain columns of each 32-row chunk."""
    B = len(A)
    nch = (B + 31) // 32
    L, U = np.eye(32 * nch, dtype=complex), np.eye(32 * nch, dtype=complex)
    U[:B, :B] = A
    for k in range(B):
        e = min(B, k + 17)
        m = U[k + 1:e, k] / U[k, k]
        L[k + 1:e, k] = m
        U[k + 1:e, k:e] -= np.outer(m, U[k, k:e])
        U[k + 1:e, k] = 0
    out = []
    for c in range(nch):
        s, lo, hi = slice(32 * c, 32 * c + 32), slice(32 * c - 16, 32 * c), slice(32 * c + 32, 32 * c + 48)
        TL, TU = np.linalg.inv(L[s, s]), np.linalg.inv(U[s, s])
        out.append((TL, -TL @ L[s, lo] if c else None, TU, -TU @ U[s, hi] if c + 1 < nch else None))
    return out


def _sweeps(F, b, dtype):
    """M^-1 b by the two sweeps, in the arithmetic of dtype."""
    nch = len(F)
    F = [[t if t is None else t.astype(dtype) for t in f] for f in F]
    x = np.zeros(32 * nch, dtype)
    x[:len(b)] = b
    for c in range(nch):
        s = slice(32 * c, 32 * c + 32)
        x[s] = F[c][0] @ x[s]
        if c:
            x[s] += F[c][1] @ x[32 * c - 16:32 * c]
    for c in range(nch - 1, -1, -1):
        s = slice(32 * c, 32 * c + 32)
        x[s] = F[c][2] @ x[s]
        if c + 1 < nch:
            x[s] += F[c][3] @ x[32 * c + 32:32 * c + 48]
    return x[:len(b)]


@pytest.mark.parametrize("ns", [27, 60, 124, 250])
def test_preconditioner_rows(tmp_path, native_lib, ns):
    """The block solves with 8 warps per block row against the FP64 ones with
    4, row by row relative to the row's value.  What FP64 sweeps leave there is
    measured on the same factors, in double against extended precision; the
    two kernels may differ by 8 times the worst row's (two errors of that kind,
    the largest of a few hundred rows each)."""
    prob, p = _problem(tmp_path, ns)
    B = 2 * (ns + 5)
    order = np.arange(B).reshape(2, -1).T.reshape(-1)      # a spline's two functions side by side
    S, Hst = O.stationary(p, DT)
    PT = (S + Hst).T.tocsr()
    s = Solver(prob, DT)
    seen = {}
    for r in range(prob.n // B):
        seen.setdefault(int(p.kappa[r]), r)                # one block row per kappa
    fac = {r: _factors(PT[r * B + order][:, r * B + order].toarray()) for r in seen.values()}
    for name, b in _vectors(prob.n // B, B, np.random.default_rng(ns)).items():
        y = {}
        for warps in (4, 8):
            s.set_precond_warps(warps)
            y[warps] = s.precond(b)
        for r, F in fac.items():
            rows = r * B + order
            ext = _sweeps(F, b[rows], np.clongdouble)
            e64 = (np.abs(_sweeps(F, b[rows], complex) - ext) / np.abs(ext)).max()
            err = (np.abs(y[8][rows] - y[4][rows]) / np.abs(y[4][rows])).max()
            assert err <= 8 * e64, (name, r, float(err), float(e64))


@pytest.mark.parametrize("n", [37, 1024, 3000])
@pytest.mark.parametrize("R,P", [(1, 1), (5, 2), (33, 4), (9, 7)])
def test_projection_of_spread_entries(native_lib, n, R, P):
    """gade_pod_project_fp64 with the entries of the basis and of the states
    spread over 24 orders of magnitude each, apart, together and opposed (so
    that every product is of one size): within 2e-15 of sum |U_i x_i|, a chunk's
    1,024 complex products in FP64 (their random walk is 64 x 2^-53 at most,
    and a lane sums only 32 of them)."""
    import torch
    from dirac_hydrogen_code_gb300 import native
    rng = np.random.default_rng(n + R + P)
    t = rng.uniform(-12, 12, n)
    z = rng.standard_normal((R, n)) + 1j * rng.standard_normal((R, n))
    w = rng.standard_normal((P, n)) + 1j * rng.standard_normal((P, n))
    for su, sx in ((t, -t), (t, t), (t, rng.uniform(-12, 12, n)), (0 * t, t)):
        U = (z * 10.0 ** su).astype(np.complex64)
        x = w * 10.0 ** sx
        Ud, xd = torch.from_numpy(U).cuda(), torch.from_numpy(x).cuda()
        sb = native.call("gade_pod_project_scratch", n, R, P)
        scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")
        coef = torch.empty(P, R, dtype=torch.complex128, device="cuda")
        native.call("gade_pod_project_fp64", n, R, Ud.data_ptr(), xd.data_ptr(), n, P, coef.data_ptr(),
                    scratch.data_ptr(), sb, 0)
        torch.cuda.synchronize()
        U64 = U.astype(np.clongdouble)
        ref, mag = x @ U64.conj().T, np.abs(x) @ np.abs(U64).T
        assert np.all(np.abs(coef.cpu().numpy() - ref) <= 2e-15 * mag)
        # a NaN reaches its own coefficients only
        xd[P - 1, n // 2] = float("nan")
        native.call("gade_pod_project_fp64", n, R, Ud.data_ptr(), xd.data_ptr(), n, P, coef.data_ptr(),
                    scratch.data_ptr(), sb, 0)
        torch.cuda.synchronize()
        c = coef.cpu().numpy()
        assert np.isnan(c[P - 1]).all()
        assert np.all(np.abs(c[:P - 1] - ref[:P - 1]) <= 2e-15 * mag[:P - 1])
