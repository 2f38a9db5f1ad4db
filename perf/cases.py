"""Performance cases of the Crank-Nicolson framework: what a user has it do,
through its public entry points, from the smallest problem to the largest.

A case is a dict of plain values.  Its ``kind`` names the entry point:

``steps``    ``native.Solver``: set a state, advance it ``steps`` Crank-Nicolson
             steps, read it back (the time loop of one pulse, restarted from a
             checkpoint inside the pulse).
``batch``    ``native.Batch``: the same for several pulses of different
             intensity at once (an intensity scan).
``apply``    ``Solver.set_time`` and four ``apply_dot_noalloc`` calls: the
             operator inside a caller's own Krylov solver.
``guess``    ``gade_learned_guess_step``: projection of the states, network and
             expansion of the learned initial guess, once per batch step.
``project``  ``gade_pod_project_fp64``: projections of training trajectories.
``train``    ``learned.MLP.train_batch``: one minibatch of the guess's training.
``eigproj``  ``gade_eigproj``: populations of the states of a batch.

The input files of a problem are generated once and kept in the temporary
directory, as a user keeps a work directory; a solver or batch (which depends
on the problem, the time step and the precision, not on the state or the
pulse's intensity) is kept between states as a user's program keeps it.
"""
import hashlib
import json
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from dirac_hydrogen_code_gb300 import native
from dirac_hydrogen_code_gb300.cn import pulse
from dirac_hydrogen_code_gb300.gen import CONFIGS, generate
from dirac_hydrogen_code_gb300.learned import MLP
from dirac_hydrogen_code_gb300.populations import E_NEG, Eigenbasis

SOL = 137.035999084
K_HIST = 4


def _problem_keys(name):
    """The sizes of one of the framework's named workloads, as case values."""
    p = CONFIGS[name]
    return dict(nsplines=p["Nsplines"], nkappa=p["Nkappa"], nmu=p["Nmu"], nl=p["Nl"], omega=p["Omega"],
                cycles=p["Cycles"], ntime=p["Ntime"], intensity=p["Intensity"])


def listed():
    small, medium, large = (_problem_keys(n) for n in ("dipole_small", "nondipole_medium", "nondipole_large"))
    return [
        # dipole workload, N = 8,400: launch and latency bound steps
        dict(name="small_steps_fp64", kind="steps", precision="fp64", tol=1e-12, steps=24, **small),
        # the benchmark's single pulse, N = 53,040, 40M operator entries
        dict(name="medium_steps_fp64", kind="steps", precision="fp64", tol=1e-12, steps=8, **medium),
        # the largest workload, N = 244,000, 342M operator entries
        dict(name="large_steps_fp64", kind="steps", precision="fp64", tol=1e-12, steps=2, **large),
        # the same pulses in mixed precision at its usual tolerance
        dict(name="medium_steps_mixed", kind="steps", precision="mixed", tol=1e-10, steps=8, **medium),
        dict(name="large_steps_mixed", kind="steps", precision="mixed", tol=1e-10, steps=6, **large),
        # intensity scans: several pulses advanced together
        dict(name="medium_batch_fp64", kind="batch", precision="fp64", tol=1e-12, steps=3, npulse=8, **medium),
        dict(name="medium_batch_mixed", kind="batch", precision="mixed", tol=1e-10, steps=4, npulse=8, **medium),
        # the operator in a caller's own solver
        dict(name="medium_apply", kind="apply", **medium),
        # per-step work of the learned guess: 8 held-out pulses of the largest workload
        dict(name="large_guess", kind="guess", n=244000, rank=128, npulse=8, hidden=256),
        # projections of the training pulses' states
        dict(name="medium_project", kind="project", n=53040, rank=128, npulse=16),
        # one minibatch of the guess's network
        dict(name="train_512", kind="train", rows=512, rank=128, hidden=256),
        # populations of a batch's states
        dict(name="medium_eigproj", kind="eigproj", npulse=8, **medium),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_problem(rng, most_kappa):
    nkappa = rng.randint(2, most_kappa)
    cycles = rng.randint(1, 4)
    return dict(nsplines=_log(rng, 20, 250), nkappa=nkappa, nmu=rng.choice([0, 0, max(2, nkappa // 2)]),
                nl=rng.choice([0, 1, rng.randint(2, 10)]), omega=float(rng.randint(10, 100)), cycles=cycles,
                ntime=500 * cycles, intensity=float(rng.choice([3, 10, 30])))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "batch", "apply", "guess", "project", "train", "eigproj"])
    if kind == "steps":
        prec = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, precision=prec, tol=rng.choice([1e-10, 1e-12]), steps=rng.randint(2, 8),
                    **_draw_problem(rng, 8))
    if kind == "batch":
        prec = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, precision=prec, tol=rng.choice([1e-10, 1e-12]), steps=rng.randint(1, 3),
                    npulse=_log(rng, 2, 12), **_draw_problem(rng, 6))
    if kind == "apply":
        return dict(kind=kind, **_draw_problem(rng, 8))
    if kind == "guess":
        return dict(kind=kind, n=_log(rng, 5000, 244000), rank=rng.randint(16, 128), npulse=_log(rng, 1, 64),
                    hidden=rng.choice([64, 128, 256]))
    if kind == "project":
        return dict(kind=kind, n=_log(rng, 5000, 200000), rank=rng.randint(16, 128), npulse=_log(rng, 1, 32))
    if kind == "train":
        return dict(kind=kind, rows=_log(rng, 32, 2048), rank=rng.randint(16, 128), hidden=rng.choice([64, 128, 256]))
    return dict(kind=kind, npulse=_log(rng, 1, 32), **_draw_problem(rng, 6))


# ---------------------------------------------------------------- problems
_PROBLEMS = {}          # work directory -> native.Problem
_HANDLE = [None, None]  # the solver or batch of the last problem: (key, handle)
_EIGEN = [None, None]


def _workdir(case):
    """The generated input files of the case's problem."""
    params = dict(Nsplines=case["nsplines"], Ntime=case["ntime"], Nkappa=case["nkappa"], Nmu=case["nmu"],
                  Nl=case["nl"], rBox=30.0, Intensity=case["intensity"], Omega=case["omega"],
                  Cycles=case["cycles"], Z=1)
    tag = hashlib.sha1(json.dumps(params, sort_keys=True).encode()).hexdigest()[:16]
    path = os.path.join(tempfile.gettempdir(), "gade_inputs_%d_%s" % (os.getuid(), tag))
    if not os.path.exists(os.path.join(path, "info.json")):
        tmp = tempfile.mkdtemp(prefix="gade_gen_")
        info = generate(params, tmp)
        with open(os.path.join(tmp, "info.json"), "w") as f:
            json.dump(info, f)
        try:
            os.rename(tmp, path)
        except OSError:                    # another process was first
            shutil.rmtree(tmp, ignore_errors=True)
    with open(os.path.join(path, "info.json")) as f:
        return path, json.load(f)


def _problem(case):
    path, info = _workdir(case)
    if path not in _PROBLEMS:
        _PROBLEMS.clear()
        _PROBLEMS[path] = native.Problem(path, info["lmax"])
    return _PROBLEMS[path]


def _dt(case):
    return case["cycles"] * 2 * math.pi / case["omega"] / case["ntime"]


def _handle(case):
    prob = _problem(case)
    key = json.dumps([prob.workdir, case["kind"], case.get("precision"), case.get("npulse")])
    if _HANDLE[0] != key:
        _HANDLE[:] = [None, None]
        if case["kind"] == "batch":
            h = native.Batch(prob, [_dt(case)] * case["npulse"], None, precision=case["precision"])
        else:
            h = native.Solver(prob, _dt(case), precision=case.get("precision", "fp64"))
        _HANDLE[:] = [key, h]
    return _HANDLE[1]


def _state(psi, nblk, kappa, rng):
    """A state inside a pulse: the ground state, and in every other block row
    a smooth radial function whose size falls over orders of magnitude."""
    X = psi.reshape(nblk, -1)
    B = X.shape[1]
    r0 = int(np.argmax(np.linalg.norm(X, axis=1)))
    g = X[r0]
    t = np.tile(np.linspace(0.0, 1.0, B // 2), 2)
    out = np.empty_like(X)
    for r in range(nblk):
        a = rng.standard_normal(4)
        f = g * (1.0 + 0.3 * sum(a[j] * np.cos((j + 1) * math.pi * t) for j in range(4))) * \
            (t + 1e-3) ** min(abs(int(kappa[r])) - 1, 3)
        size = 10.0 ** -rng.uniform(0.5, 5.0) * np.exp(2j * math.pi * rng.uniform())
        out[r] = g if r == r0 else f * (size / np.linalg.norm(f) * np.linalg.norm(g))
    return np.ascontiguousarray(out.reshape(-1))


def _pulse_in(case, rng):
    """Intensity and first step of a segment around the middle of the pulse."""
    return case["intensity"] * math.exp(rng.uniform(-0.2, 0.2)), int(case["ntime"] * rng.uniform(0.3, 0.6))


def _inputs(case, seed):
    """Host inputs of the solver cases, from the seed alone."""
    rng = np.random.default_rng(seed)
    prob = _problem(case)
    psi, _ = prob.psi0()
    nblk = int(prob.info["nblk"])
    kappa, _ = prob.blocks()
    steps = case.get("steps", 1)
    x, ft = [], []
    for _ in range(case.get("npulse", 1)):
        e0, j0 = _pulse_in(case, rng)
        x.append(_state(psi, nblk, kappa, rng))
        ft.append([pulse(e0, case["omega"], case["cycles"], (j0 + j) * _dt(case)) for j in range(steps)])
    return np.stack(x), np.stack(ft)               # [npulse, n], [npulse, steps, 6]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "batch"):
        x, ft = _inputs(case, seed)
        return dict(case=case, h=_handle(case), x=x, ft=ft)
    if kind == "apply":
        h = _handle(case)
        x, ft = _inputs(dict(case, npulse=4), seed)
        r0 = torch.from_numpy(x[::-1].copy()).cuda()
        xd = torch.from_numpy(x).cuda()
        return dict(case=case, h=h, x=xd, r0=r0, ft=ft[0, 0], y=torch.empty_like(xd),
                    dot=torch.empty(4, dtype=torch.complex128, device="cuda"))
    if kind in ("guess", "project"):
        g = _gen(seed)
        n, R, P = case["n"], case["rank"], case["npulse"]
        U = torch.view_as_complex(_randn(g, R, n, 2) / math.sqrt(2 * n))
        x = torch.view_as_complex(_randn(g, P, n, 2, dtype=torch.float64) / math.sqrt(2 * n))
        sb = native.call("gade_pod_project_scratch", n, R, P)
        st = dict(case=case, U=U, x=x, sb=sb, scratch=torch.empty(sb, dtype=torch.uint8, device="cuda"))
        if kind == "project":
            st["coef"] = torch.empty(P, R, dtype=torch.complex128, device="cuda")
            return st
        din, dh, dout = K_HIST * 2 * R + 12, case["hidden"], 2 * R
        st["hist"] = torch.view_as_complex(_randn(g, K_HIST, P, R, 2, dtype=torch.float64))
        st["ft"] = _randn(g, P, 12, dtype=torch.float64)
        st["mu_in"], st["mu_out"] = 0.1 * _randn(g, din), 0.1 * _randn(g, dout)
        st["sd_in"], st["sd_out"] = 1.0 + torch.rand(din, generator=g, device="cuda"), \
            1.0 + torch.rand(dout, generator=g, device="cuda")
        dims = [(din, dh), (dh, dh), (dh, dout)]
        st["W16"] = [(_randn(g, a, b) * math.sqrt(2.0 / a)).to(torch.bfloat16) for a, b in dims]
        st["b"] = [0.1 * _randn(g, b) for _, b in dims]
        f32, b16 = dict(dtype=torch.float32, device="cuda"), dict(dtype=torch.bfloat16, device="cuda")
        st["H"] = [torch.empty(P, dh, **f32), torch.empty(P, dh, **f32), torch.empty(P, dout, **f32)]
        st["H16"] = [torch.empty(P, dh, **b16), torch.empty(P, dh, **b16)]
        st["x16"] = torch.empty(P, din, **b16)
        st["c"] = torch.empty(P, R, dtype=torch.complex64, device="cuda")
        st["scale"] = torch.empty(P, **f32)
        st["corr"] = torch.empty(P, n, dtype=torch.complex128, device="cuda")
        p = native.LearnedGuessPlan()
        p.n, p.R, p.npulse, p.K, p.din, p.dh, p.dout = n, R, P, K_HIST, din, dh, dout
        p.U, p.hist, p.x, p.ldx = U.data_ptr(), st["hist"].data_ptr(), x.data_ptr(), n
        p.scratch, p.scratch_bytes = st["scratch"].data_ptr(), sb
        p.mu_in, p.sd_in, p.mu_out, p.sd_out = (st[k].data_ptr() for k in ("mu_in", "sd_in", "mu_out", "sd_out"))
        p.x16 = st["x16"].data_ptr()
        for i in range(3):
            p.W16[i], p.bias[i] = st["W16"][i].data_ptr(), st["b"][i].data_ptr()
        p.H1, p.H2, p.out = (t.data_ptr() for t in st["H"])
        p.H1_16, p.H2_16 = (t.data_ptr() for t in st["H16"])
        p.c, p.scale, p.corr, p.ldcorr = st["c"].data_ptr(), st["scale"].data_ptr(), st["corr"].data_ptr(), n
        p.limit = 100.0
        st["plan"] = p
        return st
    if kind == "train":
        din, dh, dout, M = K_HIST * 2 * case["rank"] + 12, case["hidden"], 2 * case["rank"], case["rows"]
        g = _gen(seed)
        mlp = MLP(din, dh, dout, max_rows=M, seed=seed)
        return dict(case=case, mlp=mlp, X=_randn(g, M, din).to(torch.bfloat16), T=_randn(g, M, dout))
    x, _ = _inputs(case, seed)
    e, xd = _eigenbasis(case), torch.from_numpy(x).cuda()
    nblk = len(e["kidx"])
    return dict(case=case, e=e, x=xd, coef=torch.empty(len(x), nblk, e["B"], dtype=torch.complex128, device="cuda"),
                cls=torch.empty(len(x), nblk, 4, dtype=torch.float64, device="cuda"))


def _eigenbasis(case):
    path, _ = _workdir(case)
    if _EIGEN[0] != path:
        kap, _ = _problem(case).blocks()
        b = Eigenbasis(path, kap)
        _EIGEN[:] = [path, dict(B=b.B, W=torch.from_numpy(b.W).cuda(), E=torch.from_numpy(b.evals).cuda(),
                                kidx=torch.from_numpy(b.block_kidx).cuda())]
    return _EIGEN[1]


# ---------------------------------------------------------------- run
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "steps":
        h = st["h"]
        h.restart(st["x"][0])
        for f in st["ft"][0]:
            h.step(f, maxit=500, tol=case["tol"])
        return h.get_x()
    if kind == "batch":
        h, P = st["h"], case["npulse"]
        for k in range(P):
            h.set_x(k, st["x"][k])
        for j in range(case["steps"]):
            h.step(st["ft"][:, j], maxit=500, tol=case["tol"])
        return [h.get_x(k) for k in range(P)]
    s = torch.cuda.current_stream().cuda_stream
    if kind == "apply":
        h, n = st["h"], st["x"].shape[1]
        h.set_time(st["ft"])
        for k in range(4):
            o = 16 * n * k
            h.apply_dot_noalloc(st["x"].data_ptr() + o, st["r0"].data_ptr() + o, st["y"].data_ptr() + o,
                                st["dot"].data_ptr() + 16 * k, s)
        return st["y"], st["dot"]
    if kind == "guess":
        native.call("gade_learned_guess_step", native.C.byref(st["plan"]), K_HIST - 1, st["ft"].data_ptr(), s)
        return st["hist"][K_HIST - 1], st["H"][2], st["c"], st["scale"], st["corr"]
    if kind == "project":
        native.call("gade_pod_project_fp64", case["n"], case["rank"], st["U"].data_ptr(), st["x"].data_ptr(),
                    case["n"], case["npulse"], st["coef"].data_ptr(), st["scratch"].data_ptr(), st["sb"], s)
        return st["coef"]
    if kind == "train":
        mlp = st["mlp"]
        loss = mlp.train_batch(st["X"], st["T"], case["rows"], 1e-3, s)
        return [loss] + list(mlp.grads) + list(mlp.params)
    e = st["e"]
    native.call("gade_eigproj", case["npulse"], len(e["kidx"]), e["B"], e["kidx"].data_ptr(), e["W"].data_ptr(),
                e["E"].data_ptr(), E_NEG, st["x"].data_ptr(), st["x"].shape[1], st["coef"].data_ptr(),
                st["cls"].data_ptr(), s)
    return st["coef"], st["cls"]


# ---------------------------------------------------------------- work
def work(case):
    """Bytes of the inputs and outputs and arithmetic of one pass.  A solver
    step counts one right-hand side and one BiCGSTAB iteration (two operator
    products, two block solves), the least it takes; an operator product two
    multiply-adds per stored entry (real entries, complex vectors)."""
    kind = case["kind"]
    if kind in ("steps", "batch", "apply", "eigproj"):
        _, i = _workdir(case)
        n, P, B = i["n"], case.get("npulse", 1), i["blkdim"]
        tables = 6 * i["lmax"] * 4 * i["blk_nnz"] * 8
        if kind == "eigproj":
            nk = 2 * case["nkappa"]
            return dict(bytes=nk * B * B * 8 + P * n * 32, flops=4.0 * P * n * B)
        product, solve = 4.0 * i["nnz_full"], 8.0 * n * 62
        if kind == "apply":
            return dict(bytes=tables + 4 * 48 * n, flops=4 * product)
        s = case["steps"]
        return dict(bytes=tables + 32 * n * P, flops=P * s * (3 * product + 2 * solve))
    if kind in ("guess", "project"):
        n, R, P = case["n"], case["rank"], case["npulse"]
        if kind == "project":
            return dict(bytes=8 * n * R + 16 * n * P + 16 * R * P, flops=8.0 * n * R * P)
        din, dh, dout = K_HIST * 2 * R + 12, case["hidden"], 2 * R
        w = din * dh + dh * dh + dh * dout
        return dict(bytes=8 * n * R + 32 * n * P + 2 * w, flops=16.0 * n * R * P + 2.0 * w * P)
    din, dh, dout, M = K_HIST * 2 * case["rank"] + 12, case["hidden"], 2 * case["rank"], case["rows"]
    w = din * dh + dh * dh + dh * dout
    return dict(bytes=28 * w + M * (2 * din + 4 * dout), flops=2.0 * M * (3 * w - din * dh))


# ---------------------------------------------------------------- exact
def _read_csr(path):
    raw = np.fromfile(path, np.uint8)
    n, nnz = (int(v) for v in raw[:8].view("<i4"))
    o = 8
    ap = raw[o:o + 4 * (n + 1)].view("<i4"); o += 4 * (n + 1)
    ai = raw[o:o + 4 * nnz].view("<i4"); o += 4 * nnz
    ax = raw[o:o + 16 * nnz].copy().view("<c16"); o += 16 * nnz
    perm = raw[o:o + 4 * n].copy().view("<i4") if len(raw) >= o + 4 * n and n else None
    m = np.zeros((n, n), complex)
    m[np.repeat(np.arange(n), np.diff(ap)), ai] = ax
    return m, perm


def _kappa(i):
    ii = i // 4
    a = int(0.5 * (math.sqrt(8.0 * ii + 1.0) - 1.0)) + 1
    return a if (i - 2.0 * a * (a - 1)) / max(4, a * 4) >= 0.5 else -a


class _Exact:
    """The operator S + H(t) and the Crank-Nicolson step as dense products."""

    def __init__(self, case):
        path, info = _workdir(case)
        rd = lambda f: _read_csr(os.path.join(path, f))  # noqa: E731
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.lmax, self.dt = info["lmax"], _dt(case)
        perm = rd("H.csr")[1]
        self.nblk, self.B = len(perm), info["blkdim"]
        self.kap = np.array([_kappa(int(p)) for p in perm], float)
        self.k = dev(self.kap)[:, None]
        self.H = [[dev(rd("H%dl%d.csr" % (u, l))[0][np.ix_(perm, perm)]) for u in (0, 1)] for l in range(self.lmax)]
        self.g = [[[dev(rd("g%da%dl%d.csr" % (q, a, l))[0]) for q in range(4)] if a % 2 != l % 2 else None
                   for a in range(6)] for l in range(self.lmax)]
        h0, s0 = [rd("h0%d.csr" % q)[0] for q in range(4)], [rd("s%d.csr" % q)[0] for q in range(3)]
        self.S, self.D, self.Pinv = {}, {}, {}
        ih = 0.5j * self.dt
        for k in sorted(set(self.kap)):
            S = s0[0] + k * s0[1] + k * k * s0[2]
            D = ih * (h0[0] + k * h0[1] + k * k * h0[2] + k ** 3 * h0[3])
            self.S[k], self.D[k] = dev(S), dev(D)
            self.Pinv[k] = dev(np.linalg.inv((S + D).T))
        self.rows = {k: torch.from_numpy(np.nonzero(self.kap == k)[0]).cuda() for k in self.S}

    def set_time(self, ft):
        c = SOL * 0.5j * self.dt
        self.pg = []
        for l in range(self.lmax):
            m = [sum(complex(c * ft[a]) * self.g[l][a][q] for a in range(6) if a % 2 != l % 2) for q in range(4)]
            # pgt: the conjugate transposes of g with the same coefficients
            t = [sum(complex(c * ft[a]) * self.g[l][a][q].conj().T for a in range(6) if a % 2 != l % 2)
                 for q in range(4)]
            self.pg.append((m, t))

    def blocks(self, M, X):
        Y = torch.empty_like(X)
        for k, r in self.rows.items():
            Y[r] = X[r] @ M[k].T
        return Y

    def parts(self, x):
        X = x.reshape(self.nblk, self.B)
        Y, kX = self.blocks(self.D, X), self.k * X
        for l in range(self.lmax):
            m, t = self.pg[l]
            a, b = self.H[l][0] @ X, self.H[l][0] @ kX
            Y += a @ m[0].T + b @ m[2].T + self.k * (a @ m[1].T + b @ m[3].T)
            a, b = self.H[l][1] @ X, self.H[l][1] @ kX
            Y += a @ t[0].T + b @ t[1].T + self.k * (a @ t[2].T + b @ t[3].T)
        return self.blocks(self.S, X).reshape(-1), Y.reshape(-1)

    def apply(self, x):
        s, h = self.parts(x)
        return s + h

    def precond(self, x):
        return self.blocks(self.Pinv, x.reshape(self.nblk, self.B)).reshape(-1)

    def solve(self, b, x):
        """BiCGSTAB inside iterative refinement, to the last digits."""
        bn = float(torch.linalg.vector_norm(b))
        last = math.inf
        for _ in range(6):
            r = b - self.apply(x)
            rn = float(torch.linalg.vector_norm(r))
            if rn < 1e-15 * bn or rn > 0.5 * last:
                break
            last = rn
            e, rr, r0, p, v = torch.zeros_like(x), r.clone(), r, torch.zeros_like(x), torch.zeros_like(x)
            rho = al = w = 1.0 + 0j
            for _ in range(12):
                rho1 = complex(torch.vdot(r0, rr))
                p = rr + (rho1 / rho) * (al / w) * (p - w * v)
                rho, y = rho1, self.precond(p)
                v = self.apply(y)
                al = rho / complex(torch.vdot(r0, v))
                s = rr - al * v
                z = self.precond(s)
                t = self.apply(z)
                w = complex(torch.vdot(t, s)) / complex(torch.vdot(t, t))
                e += al * y + w * z
                rr = s - w * t
                if float(torch.linalg.vector_norm(rr)) < max(1e-8 * rn, 1e-16 * bn):
                    break
            x = x + e
        return x

    def step(self, x, ft):
        self.set_time(ft)
        s, h = self.parts(x)
        return self.solve(s - h, x)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("steps", "batch", "apply", "eigproj"):
        x, ft = _inputs(dict(case, npulse=4) if kind == "apply" else case, seed)
        if kind == "eigproj":
            e = _eigenbasis(case)
            X = torch.from_numpy(x).cuda().reshape(len(x), -1, e["B"])
            W, E = e["W"], e["E"]
            c = torch.stack([X[:, r].conj() @ W[k].to(X.dtype) for r, k in enumerate(e["kidx"].tolist())], 1)
            p, Er = c.abs() ** 2, E[e["kidx"].long()][None]
            z = torch.zeros_like(p)
            return c, torch.stack([torch.where(m, p, z).sum(-1) for m in
                                   (Er < E_NEG, (Er >= E_NEG) & (Er < 0), Er >= 0, Er > -math.inf)], -1)
        op = _Exact(case)
        xd = [torch.from_numpy(v).cuda() for v in x]
        if kind == "apply":
            op.set_time(ft[0, 0])
            y = torch.stack([op.apply(v) for v in xd])
            return y, torch.stack([torch.vdot(xd[3 - k], y[k]) for k in range(4)])
        for k in range(len(xd)):
            for f in ft[k]:
                xd[k] = op.step(xd[k], f)
        out = [v.cpu().numpy() for v in xd]
        return out if kind == "batch" else out[0]
    st = prepare(case, seed)
    bf = lambda t: t.float().to(torch.bfloat16).double()  # noqa: E731
    if kind in ("guess", "project"):
        U = st["U"].to(torch.complex128)
        coef = st["x"] @ U.conj().T
        if kind == "project":
            return coef
        h = st["hist"].clone()
        h[K_HIST - 1] = coef
        X = torch.cat([torch.view_as_real(h[j]).reshape(case["npulse"], -1) for j in range(K_HIST - 1, -1, -1)]
                      + [st["ft"]], 1)
        a = (X - st["mu_in"].double()) / st["sd_in"].double()
        for i in range(3):
            a = bf(a) @ st["W16"][i].double() + st["b"][i].double()
            a = a.clamp(min=0) if i < 2 else a
        c = torch.view_as_complex((a * st["sd_out"].double() + st["mu_out"].double())
                                  .reshape(case["npulse"], case["rank"], 2))
        return coef, a, c, torch.ones(case["npulse"], dtype=torch.float64), c @ U
    m, X, T, M = st["mlp"], st["X"].double(), st["T"].double(), case["rows"]
    W, b = [w.double() for w in m.W], [v.double() for v in m.b]
    W16 = [bf(w) for w in W]
    H1 = (X @ W16[0] + b[0]).clamp(min=0)
    H2 = (bf(H1) @ W16[1] + b[1]).clamp(min=0)
    d = bf(H2) @ W16[2] + b[2] - T
    G3 = 2.0 * d / d.numel()
    G2 = (bf(G3) @ W16[2].T) * (H2 > 0)
    G1 = (bf(G2) @ W16[1].T) * (H1 > 0)
    grads = [X.T @ bf(G1), G1.sum(0), bf(H1).T @ bf(G2), G2.sum(0), bf(H2).T @ bf(G3), G3.sum(0)]
    params = [p for pair in zip(W, b) for p in pair]
    return [(d * d).sum(1)] + grads + [p - 1e-3 * g / (g.abs() + 1e-8) for p, g in zip(params, grads)]
