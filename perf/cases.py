"""The workloads this framework is timed on: what its users have it do, through its public entry points.

* ``steps``   a run of the model between two exchanges with the host: the seven prognostic fields go
  up from pinned memory, the model makes K steps, the fields come back (``VVMGpu.upload_prognostic``,
  ``step``, ``download_prognostic``). FP64 runs return the fields as they come back; mixed-precision
  runs write them in single precision, as their history files are.
* ``batch``   the same for an ensemble of independent cases that step together (``VVMBatch``).
* ``solve``   the elliptic equation alone, on device buffers (``VVMGpu.poisson_solve_device``).
* ``network`` the learned preconditioner's network, forward and backward, on one training pair
  (``VVMGpu.learned_eval``).

``exact`` restates the step, the solve and the network in plain torch, in 64 bits.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "2d-vector-vorticity-model_b200"))

from vvm_b200 import gpu as G  # noqa: E402
from vvm_b200 import initial_state as I  # noqa: E402

PROGNOSTIC = ("zeta", "th", "qv", "qc", "qr", "u", "w")
SOLVERS = {"spectral": G.VVM_SOLVER_SPECTRAL, "multigrid": G.VVM_SOLVER_MGPCG}
PRECISIONS = {"fp64": G.VVM_PREC_FP64, "mixed": G.VVM_PREC_MIXED}


# ------------------------------------------------------------------ the cases

def _steps(NX, NZ, dx, steps, precision="fp64", solver="spectral", init="bubble", stretched=False):
    return dict(kind="steps", NX=NX, NZ=NZ, dx=dx, steps=steps, precision=precision, solver=solver, init=init,
                stretched=stretched)


def _batch(count, steps, precision, uneven, NX=0, NZ=0):
    return dict(kind="batch", count=count, steps=steps, precision=precision, uneven=uneven, NX=NX, NZ=NZ)


def listed():
    named = {
        # the reference's own small warm bubble, many steps a call: latency and launches
        "bubble 128x64 fp64": _steps(128, 64, 200.0, 50),
        # one step an exchange, as a model that is coupled to others on the host makes it
        "coupled 512x128 fp64": _steps(512, 128, 200.0, 1, init="squall"),
        # the benchmark's grid at the reference's precision, and in mixed precision
        "bubble 2048x256 fp64": _steps(2048, 256, 100.0, 20),
        "bubble 2048x256 mixed": _steps(2048, 256, 100.0, 20, "mixed"),
        # the sheared squall line on stretched levels, dz 100 to 500 m
        "squall 1024x128 stretched fp64": _steps(1024, 128, 250.0, 20, init="squall", stretched=True),
        # the large squall line: everything comes from HBM
        "squall 8192x256 fp64": _steps(8192, 256, 100.0, 8, init="squall"),
        # an odd grid with the solver that takes any size, the default one
        "bubble 1000x101 fp64 multigrid": _steps(1000, 101, 200.0, 4, solver="multigrid"),
        # ensembles: members of one small grid, and the uneven mix of grids
        "members 48 of 256x64 mixed": _batch(48, 20, "mixed", False, 256, 64),
        "ensemble of 20 uneven mixed": _batch(20, 10, "mixed", True),
        # the elliptic solve for a caller that keeps its own model: both solvers
        "solve 2048x256 spectral": dict(kind="solve", NX=2048, NZ=256, solver="spectral"),
        "solve 1400x203 multigrid": dict(kind="solve", NX=1400, NZ=203, solver="multigrid"),
        # one training pair of the learned preconditioner, forward and backward
        "network 1024x128": dict(kind="network", NX=1024, NZ=128),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _columns(rng, lo, hi):
    """Columns the multigrid solver takes: any number whose odd factor is at most 256."""
    NX = _spread(rng, lo, hi)
    m = max(0, ((NX - 1) // 256).bit_length())
    return max(lo, NX >> m << m)


def draw(rng):
    """Another case of these ranges. In mixed precision the runs start from rest: in the sheared states the
    rounding of the first steps grows past what single-precision fields of two builds could be compared by."""
    kind = rng.choice(("steps", "steps", "steps", "steps", "batch", "solve", "network"))
    NZ = _spread(rng, 40, 256)
    dx = 200.0 if NZ <= 128 else 100.0
    if kind == "steps":
        if rng.random() < 0.2:
            NX = _columns(rng, 100, 1000)
            return _steps(NX, min(NZ, 101 * 1000 // NX), dx, rng.randint(1, 4), solver="multigrid",
                          init=rng.choice(("bubble", "squall")))
        NX = 2 ** rng.randint(7, 13)
        most = min(50, max(4, 8 * 8192 * 256 // (NX * NZ)))
        if rng.random() < 0.35:
            return _steps(NX, NZ, dx, _spread(rng, 1, min(20, most)), "mixed")
        stretched = NZ <= 128 and rng.random() < 0.25
        return _steps(NX, NZ, dx, _spread(rng, 1, most), init="squall" if stretched else rng.choice(("bubble", "squall")),
                      stretched=stretched)
    if kind == "batch":
        precision = rng.choice(("mixed", "mixed", "fp64"))
        if rng.random() < 0.5:
            return _batch(rng.randint(4, 20 if precision == "mixed" else 10), rng.randint(4, 10), precision, True)
        return _batch(rng.randint(8, 48), rng.randint(8, 20), precision, False, 2 ** rng.randint(7, 8), rng.randint(40, 64))
    if kind == "solve":
        if rng.random() < 0.5:
            return dict(kind="solve", NX=2 ** rng.randint(7, 11), NZ=NZ, solver="spectral")
        return dict(kind="solve", NX=_columns(rng, 100, 1400), NZ=min(NZ, 203), solver="multigrid")
    return dict(kind="network", NX=8 * rng.randint(16, 128), NZ=rng.randint(40, 128))


# ------------------------------------------------------------------ inputs

def _initial(NX, NZ, dx, init, stretched, seed):
    """A seeded moist state: a warm bubble or a squall line that carries a cloud with a rain shaft."""
    rng = np.random.default_rng(seed)
    xc, radius = rng.uniform(0.35, 0.65), rng.uniform(1500.0, 2500.0)
    if init == "squall":
        if stretched:
            zf = I.stretched_faces(NZ, 100.0, 100.0 + 400.0 * NZ / 128.0)
            st = I.squall_line(NX, NZ, dx, 100.0, 2.0, seed=seed, zf=zf)
        else:
            st = I.squall_line(NX, NZ, dx, dx, 1.0, seed=seed)
    else:
        st = I.warm_bubble(NX, NZ, dx, dx, 1.0, amp=rng.uniform(1.0, 3.0), radius=radius, xc_frac=xc)
    f, inner = st.fields, (slice(1, -1), slice(1, -1))
    x = (np.arange(NX + 2)[:, None] - 0.5) * dx - xc * NX * dx
    z = st.prof["z"][None, :]
    if init != "squall":
        f["th"][inner] += np.where(z <= 1000.0, rng.normal(0.0, 0.1, (NX + 2, NZ + 2)), 0.0)[inner]
    for name, most, zc, depth in (("qc", rng.uniform(1e-3, 2e-3), 2500.0, 1500.0), ("qr", rng.uniform(5e-4, 1e-3), 1500.0, 2000.0)):
        r = np.minimum(np.hypot(x / radius, (z - zc) / depth), 1.0)
        f[name][inner] = (most * 0.5 * (np.cos(np.pi * r) + 1.0))[inner]
    for name in ("th", "qc", "qr"):
        I._center2d(f[name])
    return st


def _members(case, seed):
    """The initial states of an ensemble: one grid for all, or a draw from the uneven grids."""
    sts = []
    for j in range(case["count"]):
        NX, NZ = case["NX"], case["NZ"]
        if case["uneven"]:
            pick = np.random.default_rng(1000 + j)  # the grids of an ensemble are its own, its states the seed's
            NX, NZ = int(pick.choice((256, 512, 1024, 2048))), int(pick.choice((64, 96, 128)))
        sts.append(_initial(NX, NZ, 200.0, "bubble", False, 1000 * seed + j))
    return sts


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _vorticity_rhs(case, seed):
    """A right-hand side of cal_w: vorticity dipoles of convective size, with noise at grid scale."""
    NX, NZ, dx = case["NX"], case["NZ"], 200.0 if case["NZ"] <= 128 else 100.0
    rng = np.random.default_rng(seed)
    st = I.warm_bubble(NX, NZ, dx, dx, 1.0)
    x = (np.arange(NX + 2)[:, None] - 0.5) * dx
    z = st.prof["z"][None, :]
    zeta = rng.normal(0.0, 1e-4, (NX + 2, NZ + 2))
    for _ in range(6):
        wide, deep = rng.uniform(1000.0, 3000.0), rng.uniform(800.0, 2000.0)
        d = x - rng.uniform(0.2, 0.8) * NX * dx
        zeta += rng.uniform(0.5, 2.0) * 1e-2 * d / wide * np.exp(-(d / wide) ** 2 - ((z - rng.uniform(1000.0, 6000.0)) / deep) ** 2)
    st.fields["zeta"][:] = zeta
    I._westdown2d(st.fields["zeta"])
    return st, I.poisson_rhs(st)


def _pair(case, seed, H0, NK):
    """A training pair of the network: a smooth target, and a residual of which the target and noise have equal
    parts; rows beyond the grid zero."""
    rng = np.random.default_rng(seed)
    NX = case["NX"]
    x, t = np.zeros((H0, NX), np.float32), np.zeros((H0, NX), np.float32)
    j, k = np.arange(NX)[None, :] / NX, (np.arange(NK)[:, None] + 1) / (NK + 1)
    smooth = np.zeros((NK, NX))
    for _ in range(4):
        m, n = rng.integers(1, NX // 16), rng.integers(1, NK // 8)
        smooth += rng.normal() * np.sin(np.pi * n * k) * np.cos(2 * np.pi * (m * j + rng.random()))
    t[:NK] = smooth / np.linalg.norm(smooth)
    x[:NK] = t[:NK] + rng.standard_normal((NK, NX)) / math.sqrt(NK * NX)
    return x, t


def _weights(n, seed):
    """Weights of a trained network's size: fan-in scaled."""
    rng = np.random.default_rng(seed)
    w = rng.standard_normal(n) / math.sqrt(9 * 32)
    w[:288] *= math.sqrt(32.0)
    return w.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        st = _initial(case["NX"], case["NZ"], case["dx"], case["init"], case["stretched"], seed)
        # a tighter solve than the default 1e-10 for the iterative solver: fields of two runs can be compared
        model = G.VVMGpu(st.grid, precision=PRECISIONS[case["precision"]], solver=SOLVERS[case["solver"]],
                         poisson_tol=1e-12 if case["solver"] == "multigrid" else 1e-10)
        model.upload(st)
        begin = {n: _pinned(st.fields[n].shape) for n in PROGNOSTIC}
        for n, a in begin.items():
            a.copy_(torch.from_numpy(st.fields[n]))
        end = {n: _pinned(a.shape) for n, a in begin.items()}
        s = dict(case, model=model, begin={n: a.numpy() for n, a in begin.items()}, end=end,
                 into={n: a.numpy() for n, a in end.items()})
        if case["precision"] == "mixed":
            s["history"] = {n: torch.empty(a.shape, dtype=torch.float32) for n, a in end.items()}
        return s
    if kind == "batch":
        sts = _members(case, seed)
        batch = G.VVMBatch([st.grid for st in sts], precision=PRECISIONS[case["precision"]])
        batch.upload(sts)
        sizes = [st.fields["th"].size for st in sts]
        begin, end, into = [], {n: _pinned(sum(sizes)) for n in PROGNOSTIC}, [{} for _ in sts]
        all_in = {n: _pinned(sum(sizes)) for n in PROGNOSTIC}
        at = 0
        for st, size, views in zip(sts, sizes, into):
            shape = st.fields["th"].shape
            for n in PROGNOSTIC:
                all_in[n][at:at + size] = torch.from_numpy(st.fields[n].reshape(-1))
                views[n] = end[n][at:at + size].view(shape).numpy()
            begin.append({n: all_in[n][at:at + size].view(shape).numpy() for n in PROGNOSTIC})
            at += size
        s = dict(case, batch=batch, begin=begin, end=end, into=into)
        if case["precision"] == "mixed":
            s["history"] = {n: torch.empty(a.shape, dtype=torch.float32) for n, a in end.items()}
        return s
    if kind == "solve":
        st, b = _vorticity_rhs(case, seed)
        model = G.VVMGpu(st.grid, solver=SOLVERS[case["solver"]], warm_start=False)
        model.upload(st)
        b = torch.from_numpy(b).cuda()
        return dict(case, model=model, b=b, W=torch.empty_like(b))
    st = I.warm_bubble(case["NX"], case["NZ"])
    model = G.VVMGpu(st.grid, solver=G.VVM_SOLVER_LEARNED)
    model.upload(st)
    H0, _, n = model.learned_shape()
    model.learned_weights(_weights(n, seed))
    x, t = _pair(case, seed, H0, case["NZ"] - 1)
    return dict(case, model=model, x=x, t=t)


# ------------------------------------------------------------------ one pass

def run(s):
    kind = s["kind"]
    if kind == "steps":
        s["model"].upload_prognostic(s["begin"])
        s["model"].step(s["steps"])
        s["model"].download_prognostic(s["into"])
    elif kind == "batch":
        for c, fields in zip(s["batch"].cases, s["begin"]):
            c.upload_prognostic(fields)
        s["batch"].step(s["steps"])
        for c, fields in zip(s["batch"].cases, s["into"]):
            c.download_prognostic(fields)
    elif kind == "solve":
        s["model"].poisson_solve_device(s["b"].data_ptr(), s["W"].data_ptr(), 1e-12)
        return s["W"]
    else:
        z, grad, loss = s["model"].learned_eval(s["x"], s["t"])
        return dict(z=z, grad=grad, loss=loss)
    if s["precision"] != "mixed":
        return s["end"]
    for n, a in s["end"].items():
        s["history"][n].copy_(a)
    return s["history"]


# ------------------------------------------------------------------ what a pass cannot do without

def _step_work(NX, NZ, steps, size):
    """Per step: the seven prognostic fields and the seven tendency histories read and written, the two
    eddy coefficients written; about 800 operations a cell, and the solve's two transforms."""
    cells = (NX + 2) * (NZ + 2)
    return steps * 30 * cells * size, steps * cells * (800 + 10 * math.log2(NX))


def work(case):
    kind = case["kind"]
    if kind in ("steps", "batch"):
        size = 8 if case["precision"] == "fp64" else 4
        if kind == "steps":
            grids = [(case["NX"], case["NZ"])]
        else:
            grids = [(case["NX"], case["NZ"])] * case["count"]
            if case["uneven"]:
                grids = []
                for j in range(case["count"]):
                    pick = np.random.default_rng(1000 + j)
                    grids.append((int(pick.choice((256, 512, 1024, 2048))), int(pick.choice((64, 96, 128)))))
        each = [_step_work(NX, NZ, case["steps"], size) for NX, NZ in grids]
        moved = sum(2 * 7 * (NX + 2) * (NZ + 2) * 8 for NX, NZ in grids)
        return {"bytes": sum(b for b, _ in each) + moved, "flops": sum(f for _, f in each)}
    cells = case["NX"] * (case["NZ"] - 1)
    if kind == "solve":
        return {"bytes": 2 * 8 * cells, "flops": cells * (10 * math.log2(case["NX"]) + 30)}
    pixels = case["NX"] * (-(-(case["NZ"] - 1) // 8) * 8)
    convs = 1 + 2 * (1 / 4 + 1 / 16) + 1 / 64
    return {"bytes": 3 * 4 * pixels, "flops": 3 * pixels * 2 * 9 * 32 * (32 * convs + 2)}


# ------------------------------------------------------------------ the same in 64 bits, in plain torch

class _Exact:
    """The model step in 64 bits: fields [nx][nz] with ghosts, the reference's order of operations in time
    (AB2 advection, buoyancy, negative-value fix, elliptic solve, Kessler, eddy coefficients, in-place
    diffusion, nudging)."""

    def __init__(self, st):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        g = st.grid
        self.dx, self.dt, self.nx, self.nz, self.dev = g.dx, g.dt, g.nx, g.nz, dev
        t = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.f = {n: t(st.fields[n]) for n in PROGNOSTIC}
        self.p = {n: t(st.prof[n]) for n in ("rhou", "rhow", "thvb", "pib", "pb", "lambda2", "z", "z_zeta", "thb_init")}
        self.hist = {}
        self.RKM = torch.zeros_like(self.f["th"])
        self.ubar, self.dubar = float(st.scalars["ubarTop"]), 0.0
        z, zz, nz = np.asarray(st.prof["z"]), np.asarray(st.prof["z_zeta"]), g.nz
        dc = np.empty(nz)
        dc[1:-1] = 2.0 * (z[1:-1] - zz[1:-1])
        dc[0], dc[-1] = dc[1], dc[-2]
        dw = np.empty(nz)
        dw[2:-1] = z[2:-1] - z[1:-2]
        dw[0] = dw[1] = dc[1]
        dw[-1] = dc[-2]
        across = np.ones(nz)
        zg = np.concatenate(([z[1] - dc[1]], z[1:-1], [z[-2] + dc[-2]]))
        across[1:-1] = zg[2:] - zg[:-2]
        a, h = np.ones(nz), np.ones(nz)
        if not np.allclose(dc[1:-1], g.dz, rtol=1e-9, atol=0):
            a[2:-1] = (z[2:-1] - z[1:-2]) / g.dx
            h[1:-1] = g.dx / dc[1:-1]
        self.dc, self.dw, self.across, self.h_top = t(dc), t(dw), t(across), float(h[-2])
        rhou, rhow, k = np.asarray(st.prof["rhou"]), np.asarray(st.prof["rhow"]), np.arange(2, nz - 1)
        self.up, self.dn = rhow[k] * h[k] / (a[k] * rhou[k]), rhow[k] * h[k - 1] / (a[k] * rhou[k - 1])
        self.ks = int(max([q for q in range(1, nz) if zz[q] <= 12000.0]))
        if np.allclose(dc[1:-1], g.dz, rtol=1e-9, atol=0):
            self.ks = int(12000.0 / g.dz + 1)

    @staticmethod
    def center(v):
        v[0, 1:-1], v[-1, 1:-1] = v[-2, 1:-1].clone(), v[1, 1:-1].clone()
        v[:, 0], v[:, -1] = v[:, 1].clone(), v[:, -2].clone()

    @staticmethod
    def westdown(v):
        v[0, 1:-1], v[-1, 1:-1] = v[-2, 1:-1].clone(), v[1, 1:-1].clone()
        v[:, :2] = 0.0
        v[:, -1] = 0.0

    @staticmethod
    def fix_negative(v):
        i = v[1:-1, 1:-1]
        pos, neg = i.clamp(min=0).sum(), i.clamp(max=0).sum()
        ok = (pos != 0) & (-neg <= pos)
        i.clamp_(min=0)
        i.mul_(torch.where(ok, 1.0 - (neg / pos).abs(), torch.ones_like(pos)))

    def ab2(self, name, new):
        old = self.hist.get(name, torch.zeros_like(new))
        self.hist[name] = new
        return self.dt * (1.5 * new - 0.5 * old)

    @staticmethod
    def upwind(m, m_lo, m_hi, d, d_lo, d_hi):
        """The third-order part of a flux through a face whose mass flux is m, its neighbours' m_lo and m_hi."""
        plus, minus = (lambda v: v.clamp(min=0)), (lambda v: v.clamp(max=0))
        return -(plus(m) * d - (plus(m) * plus(m_lo)).sqrt() * d_lo - minus(m) * d - (minus(m) * minus(m_hi)).sqrt() * d_hi) / 3.0

    def advect(self, q):
        u, w, rhou, rhow = self.f["u"], self.f["w"], self.p["rhou"], self.p["rhow"]
        fu, fw, mu, mw = torch.zeros_like(q), torch.zeros_like(q), rhou * u, rhow * w
        fu[1:, 1:] = mu[1:, 1:] * (q[1:, 1:] + q[:-1, 1:])
        fw[1:, 1:] = mw[1:, 1:] * (q[1:, 1:] + q[1:, :-1])
        c, k = slice(2, -2), slice(2, -2)
        dq, dk = q[1:] - q[:-1], q[:, 1:] - q[:, :-1]     # dq[i] = q[i + 1] - q[i]
        fu[c, k] += self.upwind(mu[2:-2, k], mu[1:-3, k], mu[3:-1, k], dq[1:-2, k], dq[:-3, k], dq[2:-1, k])
        fw[c, k] += self.upwind(mw[c, 2:-2], mw[c, 1:-3], mw[c, 3:-1], dk[c, 1:-2], dk[c, :-3], dk[c, 2:-1])
        self.center(fu)
        self.center(fw)
        fw[:, 0] = 0.0
        fw[:, -1] = 0.0
        d = -(fu[2:, 1:-1] - fu[1:-1, 1:-1]) / (2 * self.dx * rhou[1:-1])
        return d - (fw[1:-1, 2:] - fw[1:-1, 1:-1]) / (2 * self.dc[1:-1] * rhou[1:-1])

    def vorticity(self):
        f, p = self.f, self.p
        u, w, z, rhou, rhow = f["u"], f["w"], f["zeta"], p["rhou"], p["rhow"]
        U, W, fu, fw = (torch.zeros_like(z) for _ in range(4))
        U[1:-1, 1:-1] = 0.25 * (rhou[1:-1] * (u[2:, 1:-1] + u[1:-1, 1:-1]) + rhou[:-2] * (u[2:, :-2] + u[1:-1, :-2]))
        W[1:-1, 1:-1] = 0.25 * (rhow[2:] * (w[1:-1, 2:] + w[:-2, 2:]) + rhow[1:-1] * (w[1:-1, 1:-1] + w[:-2, 1:-1]))
        self.center(U)
        self.center(W)
        W[:, 0] = 0.0
        W[:, -1] = 0.0
        fu[:-1, 1:-1] = U[:-1, 1:-1] * (z[1:, 1:-1] + z[:-1, 1:-1])
        fw[:-1, 1:-1] = W[:-1, 1:-1] * (z[:-1, 2:] + z[:-1, 1:-1])
        c, dq, dk = slice(2, -2), z[1:] - z[:-1], z[:, 1:] - z[:, :-1]
        fu[c, c] += self.upwind(U[2:-2, c], U[1:-3, c], U[3:-1, c], dq[2:-1, c], dq[1:-2, c], dq[3:, c])
        fw[c, c] += self.upwind(W[c, 2:-2], W[c, 1:-3], W[c, 3:-1], dk[c, 2:-1], dk[c, 1:-2], dk[c, 3:])
        self.center(fu)
        self.center(fw)
        fw[:, 0] = 0.0
        fw[:, -1] = 0.0
        k = slice(2, -1)
        d = -(fu[1:-1, k] - fu[:-2, k]) / (2 * self.dx * rhow[k]) - (fw[1:-1, k] - fw[1:-1, 1:-2]) / (2 * self.dw[k] * rhow[k])
        new = z.clone()
        new[1:-1, k] += self.ab2("zeta", d)
        thv = f["th"] * (1 + 0.608 * f["qv"]) / p["thvb"]
        load = f["qc"] + f["qr"]
        pairs = [0.5 * (v[1:] - v[:-1])[:-1] for v in (thv, load)]
        b = [v[:, 2:-1] + v[:, 1:-2] for v in pairs]
        new[1:-1, k] += self.ab2("buoyancy", 9.80665 / rhow[k] / self.dx * (b[0] - b[1]))
        self.westdown(new)
        return new

    def sediment(self):
        q, rhow = self.f["qr"], self.p["rhow"]
        fw = torch.zeros_like(q)
        s = q[1:-1, 1:-1] + q[1:-1, :-2]
        fall = 36.34 * (0.5e-3 * rhow[1:-1] * s) ** 0.1346 * (rhow[1:-1] / rhow[1]) ** -0.5
        fw[1:-1, 1:-1] = rhow[1:-1] * fall * s
        self.center(fw)
        fw[:, 0] = 0.0
        fw[:, -1] = 0.0
        return (fw[1:-1, 2:] - fw[1:-1, 1:-1]) / (2 * self.dc[1:-1] * self.p["rhou"][1:-1])

    def top_wind(self):
        u, w, K, rhou, rhow = self.f["u"], self.f["w"], self.RKM, self.p["rhou"], self.p["rhow"]
        i, l = slice(1, -1), slice(0, -2)
        mean = lambda v: float(v.mean())  # noqa: E731
        down = mean(0.25 * (rhou[-2] * u[i, -2] + rhou[-3] * u[i, -3]) * (w[i, -2] + w[l, -2]))
        up = mean(rhow[-1] * 0.25 * (K[i, -1] + K[i, -2] + K[l, -1] + K[l, -2]) * (u[i, -1] - u[i, -2]) / self.dw[-1])
        dn = mean(rhow[-2] * 0.25 * (K[i, -2] + K[i, -3] + K[l, -2] + K[l, -3])
                  * ((w[i, -2] - w[l, -2]) / self.dx + (u[i, -2] - u[i, -3]) / self.dw[-2]))
        d = (-down + up - dn) / float(self.dc[-2] * rhou[-2])
        new = self.ubar + self.dt * (1.5 * d - 0.5 * self.dubar)
        self.dubar = d
        return new

    def wind(self, zeta, top):
        u, w, rhou, rhow, nz = self.f["u"], self.f["w"], self.p["rhou"], self.p["rhow"], self.nz
        b = (rhow[2:-1] ** 2 * (zeta[2:, 2:-1] - zeta[1:-1, 2:-1]) * self.dx).T.contiguous()
        w[1:-1, 2:-1] = (solve_columns(b, self.up, self.dn) / rhow[2:-1, None]).T
        self.westdown(w)
        h = rhow[-2] * w[1:-1, -2] / rhou[-2] * self.dx * self.h_top
        h = h - h.mean()
        x = (torch.cumsum(h, 0) - h) / self.dx
        u[1:-1, -2] = x - x.mean() + top
        part = -((w[1:-1, 2:-1] - w[:-2, 2:-1]) / self.dx - rhow[2:-1] * zeta[1:-1, 2:-1]) * self.dw[2:-1]
        u[1:-1, 1:-2] = part.flip(1).cumsum(1).flip(1) + u[1:-1, -2:-1]
        self.center(u)

    def kessler(self, th, qv, qc, qr):
        i, rho, pi = (slice(1, -1), slice(1, -1)), self.p["rhou"][1:-1], self.p["pib"][1:-1]
        T, v, c, r = th[i].clone(), qv[i].clone(), qc[i].clone(), qr[i].clone()
        plus = lambda x: x.clamp(min=0)  # noqa: E731
        auto = torch.minimum(plus(0.001 * (plus(c) - 0.001)) * self.dt, plus(c))
        c, r = c - auto, r + auto
        acc = torch.minimum(2.2 * plus(c) * plus(r) ** 0.875 * self.dt, plus(c))
        c, r = c - acc, r + acc
        scale = 380.0 / (pi ** (1003.5 / 287.0) * 1e5)
        qvs = scale * torch.exp(17.27 * (pi * T - 273.0) / (pi * T - 36.0))
        rr = 1e-3 * rho * plus(r)
        rate = (1.6 + 124.9 * rr ** 0.2046) * plus(1.0 - plus(v) / qvs) * rr ** 0.525
        rate = rate / ((5.4e5 + 2.55e6 / (1e-2 * self.p["pb"][1:-1] * qvs)) * 1e-3 * rho)
        ev = torch.minimum(plus(r), plus(rate * self.dt))
        r, v, T = r - ev, v + ev, T - 2.5e6 * ev / (1003.5 * pi)
        qvs = scale * torch.exp(17.27 * (pi * T - 273.0) / (pi * T - 36.0))
        C = (v - qvs) / (1 + qvs * (17.27 * 237.0 * 2.5e6) / (1003.5 * (T * pi - 36.0) ** 2))
        C = torch.where((C < 0) & (C.abs() > c), -c, C)
        th[i], qv[i], qc[i], qr[i] = T + 2.5e6 / (1003.5 * pi) * C, v - C, c + C, r

    def eddies(self, th):
        u, w, dx, i, lo, hi = self.f["u"], self.f["w"], self.dx, slice(1, -1), slice(0, -2), slice(2, None)
        R = 0.5 * ((w[hi, hi] + w[hi, i]) - (w[lo, hi] + w[lo, i])) / (2 * dx)
        R = R + 0.5 * ((u[hi, hi] + u[i, hi]) - (u[hi, lo] + u[i, lo])) / self.across[i]
        rot = ((u[hi, i] - u[i, i]) / dx + (w[i, hi] - w[i, i]) / self.dc[i]) ** 2
        S2 = R ** 2 + 2 * rot
        Ri = 9.80665 / th[i, i] * (th[i, hi] - th[i, lo]) / self.across[i] / S2
        low, mid = Ri < 0, (Ri > 0) & (Ri < 0.25)
        base, p4 = self.p["lambda2"][i] * S2.sqrt(), (1 - 4 * Ri) ** 4
        zero, most = torch.zeros_like(base), (0.8 * dx * self.dc[i] / self.dt).expand_as(base)
        km = torch.where(low, base * (1 - 16 * Ri).clamp(min=0).sqrt(), torch.where(mid, base * p4, zero))
        kh = torch.where(low, base * 1.4 * (1 - 40 * Ri).clamp(min=0).sqrt(), torch.where(mid, base * 1.4 * (1 - 1.2 * Ri) * p4, zero))
        out = []
        for K in (km, kh):
            full = torch.zeros_like(th)
            full[i, i] = torch.minimum(K.clamp(min=10.0), most)
            self.center(full)
            out.append(full)
        return out

    def diffuse(self, v, K, vorticity):
        """The in-place sweep v'(i, k) of v, v'(i-1, k) and v'(i, k-1): the recurrence's fixed point."""
        i, lo, hi, p, dx2 = slice(1, -1), slice(0, -2), slice(2, None), self.p, self.dx ** 2
        rhou, rhow, dc, dw = p["rhou"], p["rhow"], self.dc, self.dw
        if vorticity:
            R, L = 0.5 * (K[i, i] + K[i, lo]), 0.5 * (K[lo, i] + K[lo, lo])
            U = rhou[i] * 0.5 * (K[i, i] + K[lo, i]) / (rhow[i] * dw[i] * dc[i])
            D = rhou[lo] * 0.5 * (K[i, lo] + K[lo, lo]) / (rhow[i] * dw[i] * dc[lo])
        else:
            R, L = 0.5 * (K[hi, i] + K[i, i]), 0.5 * (K[i, i] + K[lo, i])
            U = rhow[hi] * 0.5 * (K[i, hi] + K[i, i]) / (rhou[i] * dc[i] * dw[hi])
            D = rhow[i] * 0.5 * (K[i, i] + K[i, lo]) / (rhou[i] * dc[i] * dw[i])
        R, L, U, D = (self.dt * x for x in (R / dx2, L / dx2, U, D))
        old = v[i, i] + R * (v[hi, i] - v[i, i]) - L * v[i, i] + U * (v[i, hi] - v[i, i]) - D * v[i, i]
        for _ in range(400):
            before = v[i, i].clone()
            v[i, i] = old + L * v[lo, i] + D * v[i, lo]
            if torch.equal(before, v[i, i]):
                break

    def nudge(self, v, height, rate, toward):
        ks, nz = self.ks, self.nz
        if ks >= nz - 1:
            return
        z, z0 = self.p[height], self.p[height][nz - 1 - ks]
        c = self.dt * rate * (z[ks:-1] - z0) / (z[-1] - z0)
        v[1:-1, ks:-1] -= c * (v[1:-1, ks:-1] - toward[ks:-1])

    def step(self):
        f = self.f
        zeta, new = self.vorticity(), {}
        for n in ("th", "qv", "qc", "qr"):
            v = f[n].clone()
            v[1:-1, 1:-1] += self.ab2(n, self.advect(f[n]))
            if n == "qr":
                v[1:-1, 1:-1] += self.ab2("fall", self.sediment())
            if n != "th":
                self.fix_negative(v)
            self.center(v)
            new[n] = v
        top = self.top_wind()
        self.wind(zeta, top)
        self.kessler(*(new[n] for n in ("th", "qv", "qc", "qr")))
        for n in ("qv", "qc", "qr"):
            self.fix_negative(new[n])
        for v in new.values():
            self.center(v)
        # means of the advanced fields replace the base profiles of the next step's buoyancy
        self.RKM, RKH = self.eddies(new["th"])
        self.diffuse(zeta, self.RKM, True)
        for v in new.values():
            self.diffuse(v, RKH, False)
        self.nudge(new["th"], "z", 1.0 / 3600.0, self.p["thb_init"])
        self.nudge(zeta, "z_zeta", 1.0 / 360.0, torch.zeros_like(self.p["z"]))
        thvb = new["th"][1:-1].mean(0) * (1 + 0.608 * new["qv"][1:-1].mean(0))
        thvb[0], thvb[-1] = thvb[1].clone(), thvb[-2].clone()
        self.p["thvb"], self.ubar = thvb, top
        f.update(new, zeta=zeta)


def solve_columns(b, up, dn):
    """x[k][i] of x[i-1] + x[i+1] - 2 x + up (x[k+1] - x) + dn (x[k-1] - x) = b, periodic in i, zero beyond k:
    Fourier modes in i, one tridiagonal system in k for each."""
    NK, NX = b.shape
    r = torch.fft.rfft(b, dim=1)
    lam = -4.0 * torch.sin(torch.pi * torch.arange(r.shape[1], dtype=torch.float64, device=b.device) / NX) ** 2
    cp, x = [], []
    for k in range(NK):
        den = lam - (up[k] + dn[k]) - (dn[k] * cp[-1] if k else 0.0)
        cp.append((up[k] if k < NK - 1 else 0.0) / den)
        x.append((r[k] - (dn[k] * x[-1] if k else 0.0)) / den)
    for k in range(NK - 2, -1, -1):
        x[k] = x[k] - cp[k] * x[k + 1]
    return torch.fft.irfft(torch.stack(x), n=NX, dim=1)


def _exact_fields(st, steps):
    m = _Exact(st)
    for _ in range(steps):
        m.step()
    return {n: m.f[n].cpu() for n in PROGNOSTIC}


def _exact_network(case, seed):
    NX, NK = case["NX"], case["NZ"] - 1
    H0, C = -(-NK // 8) * 8, 32
    st = I.warm_bubble(NX, case["NZ"])
    x, t = (torch.tensor(a, dtype=torch.float64) for a in _pair(case, seed, H0, NK))
    params = torch.tensor(_weights(2 * 9 * C + 6 * 9 * C * C, seed), dtype=torch.float64, requires_grad=True)
    F = torch.nn.functional

    def conv(a, w, cin, cout):
        a = F.pad(F.pad(a[None], (1, 1, 0, 0), mode="circular"), (0, 0, 1, 1))
        return F.conv2d(a, w.reshape(3, 3, cin, cout).permute(3, 2, 0, 1))[0]

    pool = lambda a: F.avg_pool2d(a[None], 2)[0]  # noqa: E731
    twice = lambda a: a.repeat_interleave(2, 1).repeat_interleave(2, 2)  # noqa: E731
    w = params[9 * C:-9 * C].reshape(6, 9, C, C)
    h = [conv(x[None], params[:9 * C], 1, C)]
    for j in range(3):
        h.append(conv(pool(h[-1]), w[j], C, C))
    g = h[3]
    for j in range(3):
        g = conv(twice(g) + h[2 - j], w[3 + j], C, C)
    z = conv(g, params[-9 * C:], C, 1)[0]
    z = torch.cat((z[:NK], torch.zeros(H0 - NK, NX, dtype=torch.float64)))
    rhou, rhow, k = st.prof["rhou"], st.prof["rhow"], np.arange(2, NK + 2)
    cx, ru, rd = 1 / rhow[k], 1 / rhou[k], 1 / rhou[k - 1]
    s = 1 / np.sqrt(2 * cx + ru + rd)
    cx, ru, rd = (torch.tensor(v)[:, None] for v in (cx * s * s, ru[:-1] * s[:-1] * s[1:], rd[1:] * s[1:] * s[:-1]))

    def dot(a, b):
        """The energy product of the scaled operator."""
        a, b = a[:NK], b[:NK]
        y = b - cx * (b.roll(1, 1) + b.roll(-1, 1))
        return (a * y).sum() - (a[:-1] * ru * b[1:]).sum() - (a[1:] * rd * b[:-1]).sum()

    loss = 1 - dot(z, t) ** 2 / (dot(z, z) * dot(t, t))
    grad, = torch.autograd.grad(loss, params)
    return dict(z=z.detach(), grad=grad, loss=float(loss.detach()))


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        return _exact_fields(_initial(case["NX"], case["NZ"], case["dx"], case["init"], case["stretched"], seed), case["steps"])
    if kind == "batch":
        each = [_exact_fields(st, case["steps"]) for st in _members(case, seed)]
        return {n: torch.cat([f[n].reshape(-1) for f in each]) for n in PROGNOSTIC}
    if kind == "solve":
        st, b = _vorticity_rhs(case, seed)
        rhou, rhow, k = st.prof["rhou"], st.prof["rhow"], np.arange(2, case["NZ"] + 1)
        b = torch.from_numpy(b).reshape(case["NZ"] - 1, case["NX"])
        return solve_columns(b, rhow[k] / rhou[k], rhow[k] / rhou[k - 1]).reshape(-1)
    return _exact_network(case, seed)
