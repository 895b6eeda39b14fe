"""Workloads whose time is followed: what a program that uses this package has it compute.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges. ``prepare`` makes what a program
holds before the call (a lattice at rest, an ensemble, a network with its training set), ``run`` makes
one pass through the public entry points and returns everything that pass computes for its caller,
``work`` states the bytes and operations of a pass and ``exact`` computes the same outputs in 64 bits
with plain torch (no code of this package).
"""
import math

import numpy as np
import torch

from lbm_solver_3d_b200.ensemble import Ensemble
from lbm_solver_3d_b200.mlp import MLP, NPARAMS
from lbm_solver_3d_b200.params import Params
from lbm_solver_3d_b200.solver import HostFields, Solver
from lbm_solver_3d_b200.workloads import SLIT_DECK, ensemble_members

WIDTH = {"fp64": 8, "fp32": 4, "fp16": 2}
SQ_KEYS = ("X", "e", "U", "W", "Fh", "Th", "Fc", "Tc", "Fw")


# ---- the cases -----------------------------------------------------------------------------------
def lattice(name, nx, ny, nz, precision, steps, walls="", radius=0.0, b1=0.0, tau=1.0, fx=0.0, planar=True):
    """One lattice advanced `steps` time steps, then read: its fields, and with a squirmer (radius > 0)
    its state and trajectory rows."""
    return {"name": name, "kind": "lattice", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "steps": steps,
            "walls": walls, "radius": radius, "b1": b1, "tau": tau, "fx": fx, "planar": planar}


def listed():
    return [
        # the reference's tutorial duct, the smallest lattice anybody runs: one print interval, then the profile
        lattice("duct_4x34x34_fp64", 4, 34, 34, "fp64", 500, walls="yz", tau=0.8, fx=1e-6),
        # the tutorial's channel deck (64x34x32, R = 4) in the plain form: a few trajectory intervals
        lattice("channel_64x34x32_fp64", 64, 34, 32, "fp64", 400, walls="y", radius=4.0, b1=0.015),
        # the slit-channel workload in the production form
        lattice("slit_128x64x64_fp32", 128, 64, 64, "fp32", 400, walls="y", radius=6.0, b1=1.5e-3),
        # the same deck driven call by call, as a program with its own time loop does it
        dict(lattice("stepwise_64x34x32_fp64", 64, 34, 32, "fp64", 20, walls="y", radius=4.0, b1=0.015),
             kind="stepwise"),
        # the precision and roofline lattice in its three storage forms
        lattice("bulk_256x128x128_fp64", 256, 128, 128, "fp64", 200, radius=8.0, b1=1e-3, tau=0.9, planar=False),
        lattice("bulk_256x128x128_fp32", 256, 128, 128, "fp32", 200, radius=8.0, b1=1e-3, tau=0.9, planar=False),
        lattice("bulk_256x128x128_fp16", 256, 128, 128, "fp16", 200, radius=8.0, b1=1e-3, tau=0.9, planar=False),
        # odd extents, walls and a body force: nothing a multiple of anything
        lattice("ragged_149x97x83_fp32", 149, 97, 83, "fp32", 200, walls="y", radius=6.5, b1=2e-3, fx=5e-7),
        # the parameter sweep: all trajectories of 256 slit channels of uneven sizes, in FP32 storage
        {"name": "sweep_256_fp32", "kind": "ensemble", "members": 256, "precision": "fp32", "steps": 60, "fields": False},
        # a smaller sweep in FP16 storage
        {"name": "sweep_64_fp16", "kind": "ensemble", "members": 64, "precision": "fp16", "steps": 60, "fields": False},
        # one epoch of the surrogate network's training (Surrogate.fit's batch and rate)
        {"name": "train_65536_bf16", "kind": "train", "bf16": True, "n": 65536, "batch": 512},
        # the surrogate evaluated over a large sweep of states
        {"name": "forward_250001_bf16", "kind": "forward", "bf16": True, "n": 250001},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["duct", "lattice", "lattice", "lattice", "stepwise", "ensemble", "train", "forward"])
    prec = rng.choice(["fp64", "fp32", "fp32", "fp16"])
    if kind == "duct":
        c = lattice("", _log(rng, 4, 64), rng.randint(12, 66), rng.randint(12, 66), rng.choice(["fp64", "fp64", "fp32"]),
                    rng.randint(150, 600), walls=rng.choice(["y", "yz"]), tau=0.8, fx=rng.choice([1e-6, 4e-6]))
    elif kind in ("lattice", "stepwise"):
        r = round(rng.uniform(3.0, 8.0), 2)
        lo = int(2 * r) + 12
        big = 100 if kind == "stepwise" else 384
        nx, ny, nz = (max(lo, _log(rng, 24, n)) for n in (big, min(big, 128), min(big, 128)))
        if rng.random() < 0.5:   # the sizes that decks tend to have
            nx = max(32, nx // 32 * 32)
        walls = rng.choice(["y", "y", "", "yz"])
        c = lattice("", nx, ny, nz, prec, rng.randint(80, 400), walls=walls, radius=r, b1=rng.choice([1e-3, 4e-3, 0.015]),
                    tau=rng.choice([0.8, 0.9, 1.0]), fx=rng.choice([0.0, 0.0, 5e-7]), planar=walls != "")
        if kind == "stepwise":
            c.update(kind="stepwise", steps=rng.randint(5, 40))
    elif kind == "ensemble":
        n = _log(rng, 2, 128)
        c = {"kind": "ensemble", "members": n, "precision": prec, "steps": rng.randint(50, 120), "fields": n <= 6}
    elif kind == "train":
        c = {"kind": "train", "bf16": rng.random() < 0.6, "n": _log(rng, 2000, 150000), "batch": rng.choice([128, 256, 500, 512, 1024])}
    else:
        c = {"kind": "forward", "bf16": rng.random() < 0.6, "n": _log(rng, 1, 1000000)}
    c.pop("name", None)
    return c


# ---- inputs and state ----------------------------------------------------------------------------
def deck(case, seed):
    """The deck of a lattice: the case's sizes, and from the seed what differs between one user's runs
    (drive, swimming mode, start and orientation)."""
    r = np.random.default_rng([7, int(seed)])
    p = Params()
    p.update(nx=case["nx"], ny=case["ny"], nz=case["nz"], walls_y=int("y" in case["walls"]),
             walls_z=int("z" in case["walls"]), tau=case["tau"], fx=case["fx"] * float(r.uniform(0.5, 2.0)),
             precision=case["precision"], traj_every=50, steps=10000)
    if case["radius"] > 0:
        g = r.standard_normal(3)
        g /= np.linalg.norm(g)
        a = math.radians(float(r.uniform(-30.0, 30.0)))
        if case["planar"]:
            g = np.array([math.cos(a), math.sin(a), 0.0])
        c = [0.5 * (n - 1) + float(r.uniform(-1.5, 1.5)) for n in (case["nx"], case["ny"], case["nz"])]
        p.update(squirmer=1, radius=case["radius"], b1=case["b1"], beta=float(r.uniform(-3.0, 3.0)),
                 planar=int(case["planar"]), x0=c[0], y0=c[1], z0=c[2], ex=float(g[0]), ey=float(g[1]), ez=float(g[2]))
    p.validate()
    return p


def members(case, seed):
    """The sweep's channels: sizes of the 256-member workload, swimming modes and angles from the seed."""
    r = np.random.default_rng([11, int(seed)])
    ps = ensemble_members(256)[: case["members"]]
    for p in ps:
        p.update(beta=float(r.uniform(-5.0, 5.0)), angle=float(r.uniform(-30.0, 30.0)), precision=case["precision"], **SLIT_DECK)
    return ps


def states(n, seed):
    """(h/a, theta, beta, H/a) as the sweeps meet them, and a smooth velocity as target."""
    r = np.random.default_rng([13, int(seed)])
    H = r.uniform(6.0, 23.0, n)
    x = np.stack([1.2 + r.uniform(0, 1, n) * (H - 2.4), r.uniform(-0.6, 0.6, n), r.uniform(-5, 5, n), H], 1)
    x = (x - x.mean(0)) / (x.std(0) + 1e-12) if n > 1 else x / 10.0
    y = np.stack([np.cos(x[:, 1]) + 0.1 * x[:, 2] / (1 + x[:, 0] ** 2), np.sin(x[:, 1]) - 0.05 * x[:, 2], 0.2 * np.tanh(x[:, 0] * x[:, 2])], 1)
    return x.astype(np.float32), y.astype(np.float32)


def weights(seed):
    """Network parameters as a fresh network has them: uniform in +-1/sqrt(fan-in)."""
    r = np.random.default_rng([17, int(seed)])
    parts = [(64 * 4, 4), (64, 4), (64 * 64, 64), (64, 64), (64 * 64, 64), (64, 64), (3 * 64, 64), (3, 64)]
    return np.concatenate([r.uniform(-f ** -0.5, f ** -0.5, n) for n, f in parts]).astype(np.float32)


def prepare(case, seed):
    k = case["kind"]
    if k in ("lattice", "stepwise"):
        s = Solver(deck(case, seed))
        out = None
        if s.N > 200000:   # large fields are read into page-locked buffers the program keeps
            out = HostFields(s.N)
            out.flag, out.rho, out.u = (torch.empty(k * s.N, dtype=t, pin_memory=True).numpy()
                                        for k, t in ((1, torch.uint8), (1, torch.float64), (3, torch.float64)))
        return {"case": case, "s": s, "out": out}
    if k == "ensemble":
        return {"case": case, "e": Ensemble(members(case, seed))}
    net = MLP(bf16=case["bf16"], params=weights(seed))
    x, y = states(case["n"], seed)
    st = {"case": case, "net": net, "x": x}
    if k == "train":
        net.set_data(x, y)
        st["order"] = np.random.default_rng([19, int(seed)]).permutation(case["n"]).astype(np.int32)
    return st


def _read(s, out, rows=True):
    flag, rho, u = s.fields_into(out) if out is not None else s.fields()
    r = {"flag": flag, "rho": rho, "u": u}
    if s.params.squirmer:
        q = s.squirmer()
        r["squirmer"] = np.stack([q[k] for k in SQ_KEYS])
        if rows:
            r["rows"] = s.traj_rows(4096)
    return r


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "lattice":
        state["s"].run(case["steps"])
        return _read(state["s"], state["out"])
    if k == "stepwise":
        s = state["s"]
        for _ in range(case["steps"]):
            s.step()
            s.advance_squirmer()
            if s.t % s.params.massCorrectionEvery == 0:
                s.correct_mass()
        return _read(s, state["out"], rows=False)
    if k == "ensemble":
        e = state["e"]
        e.run(case["steps"])
        ms = [e.member(i) for i in range(len(e))]
        r = {"rows": np.concatenate([m.traj_rows(4096) for m in ms]),
             "squirmers": np.stack([[q[n] for n in SQ_KEYS] for q in (m.squirmer() for m in ms)])}
        if case["fields"]:
            r["fields"] = [dict(zip(("flag", "rho", "u"), m.fields())) for m in ms]
        return r
    if k == "train":
        loss = state["net"].train_epoch(state["order"], case["batch"], 2e-3)
        return {"loss": float(loss), "params": state["net"].params()}
    return state["net"].forward(state["x"])


def work(case):
    k = case["kind"]
    if k in ("lattice", "stepwise"):
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 2.0 * 19 * WIDTH[case["precision"]] * n * case["steps"] + 33.0 * n, "flops": 260.0 * n * case["steps"]}
    if k == "ensemble":
        n = sum(p.ncells for p in ensemble_members(256)[: case["members"]])
        return {"bytes": 2.0 * 19 * WIDTH[case["precision"]] * n * case["steps"], "flops": 260.0 * n * case["steps"]}
    macs = 4 * 64 + 64 * 64 * 2 + 64 * 3
    if k == "train":
        steps = -(-case["n"] // case["batch"])
        return {"bytes": case["n"] * 32.0 + steps * 6.0 * 4 * NPARAMS, "flops": 6.0 * macs * case["n"]}
    return {"bytes": case["n"] * 28.0, "flops": 2.0 * macs * case["n"]}


# ---- the same results in 64 bits -----------------------------------------------------------------
CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1]
CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1]
C = np.stack([CX, CY, CZ], 1)
OPP = np.array([0] + [i + 1 if i % 2 else i - 1 for i in range(1, 19)])
WT = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


class Plain64:
    """D3Q19 two-relaxation-time steps with Guo forcing, halfway bounce-back and one squirmer, in plain torch."""

    def __init__(self, p, u_every):
        self.p, self.u_every = p, u_every
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.n = np.array([p.NX, p.NY, p.NZ])
        self.wall = np.array([False, bool(p.wallsY), bool(p.wallsZ)])
        sh = (p.NZ, p.NY, p.NX)
        t = lambda v: torch.tensor(np.asarray(v), dtype=torch.float64, device=self.dev)  # noqa: E731
        self.w, self.c = t(WT), t(C)
        self.f = self.w.view(19, 1, 1, 1).expand(19, *sh).clone()
        self.rho = torch.ones(sh, dtype=torch.float64, device=self.dev)
        self.u = torch.zeros(sh + (3,), dtype=torch.float64, device=self.dev)
        flag = np.zeros(sh, np.uint8)
        if p.wallsY:
            flag[:, [0, -1], :] = 1
        if p.wallsZ:
            flag[[0, -1]] = 1
        self.F = np.array([p.Fx, p.Fy, p.Fz])
        self.om = (1 / p.tau, 1 / (0.5 + p.Lambda / (p.tau - 0.5)))
        self.t, self.rows, self.sq = 0, [], bool(p.squirmer)
        if self.sq:
            self.R = p.R
            self.X = np.array([c if c >= 0 else 0.5 * (m - 1) for c, m in zip((p.x0, p.y0, p.z0), self.n)], float)
            a = math.radians(p.angle)
            e = np.array(p.orientation if p.orientation is not None else (math.cos(a), math.sin(a), 0.0), float)
            self.e = e / np.linalg.norm(e)
            self.U, self.W, self.Fh, self.Th, self.Fc, self.Tc, self.Fw = (np.zeros(3) for _ in range(7))
            self.M = p.rhoP * 4 / 3 * math.pi * p.R ** 3
            self.I = 0.4 * self.M * p.R ** 2
            self.FS = 6 * math.pi * (p.tau - 0.5) / 3 * p.R * (2 * p.B1 / 3)
            for z, y, x in self.changes(flag)[0]:
                flag[z, y, x] = 2
        self.set_flag(flag)

    def offset(self, pts):   # pts (..., 3) as x, y, z
        r = pts - self.X
        per = ~self.wall
        k = np.sign(r) * np.floor(np.abs(r) / self.n + 0.5)
        return np.where(per, r - self.n * k, r)

    def changes(self, flag):
        """(covered, uncovered) nodes in the box of the sphere, each in z, y, x order."""
        lo = np.floor(self.X - self.R).astype(int) - 2
        hi = np.ceil(self.X + self.R).astype(int) + 2
        if self.wall[1]:
            lo[1], hi[1] = max(0, lo[1]), min(self.n[1] - 1, hi[1])
        zz, yy, xx = np.meshgrid(*[np.arange(lo[d], hi[d] + 1) % self.n[d] for d in (2, 1, 0)], indexing="ij")
        r = self.offset(np.stack([xx, yy, zz], -1).astype(float))
        inside = r[..., 0] * r[..., 0] + r[..., 1] * r[..., 1] + r[..., 2] * r[..., 2] < self.R * self.R
        fl = flag[zz, yy, xx]
        ch = (fl != 1) & (inside != (fl == 2))
        z, y, x = zz[ch], yy[ch], xx[ch]
        return list(zip(z.tolist(), y.tolist(), x.tolist())), inside[ch]

    def set_flag(self, flag):
        self.flag = flag
        fl = torch.tensor(flag, device=self.dev)
        self.fluid = fl == 0
        di, ni, ty = [], [], []
        for i in range(1, 19):   # target n + c_i is solid
            tgt = torch.roll(fl, (-CZ[i], -CY[i], -CX[i]), (0, 1, 2))
            k = torch.nonzero((self.fluid & (tgt != 0)).view(-1)).view(-1)
            di.append(torch.full_like(k, i)); ni.append(k); ty.append(tgt.reshape(-1)[k])
        self.di, self.ni, ty = torch.cat(di), torch.cat(ni), torch.cat(ty)
        self.part = torch.nonzero(ty == 2).view(-1)
        self.oi = torch.tensor(OPP, device=self.dev)[self.di]

    def step(self, last):
        f, w, om = self.f, self.w, self.om
        rho = f.sum(0)
        m = [(torch.einsum("i,izyx->zyx", self.c[:, d], f) + 0.5 * self.F[d]) / rho for d in range(3)]
        self.rho = torch.where(self.fluid, rho, self.rho)
        if last or self.u_every:
            self.u = torch.where(self.fluid.unsqueeze(-1), torch.stack(m, -1), self.u)
        usq = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
        uF = sum(m[d] * self.F[d] for d in range(3))
        post = torch.empty_like(f)
        gP, gM = 1 - 0.5 * om[0], 1 - 0.5 * om[1]
        post[0] = f[0] - om[0] * (f[0] - WT[0] * rho * (1 - 1.5 * usq)) - gP * WT[0] * 3 * uF
        for i in range(1, 19, 2):
            cu = sum(int(C[i, d]) * m[d] for d in range(3) if C[i, d])
            cF = float(C[i] @ self.F)
            A = om[0] * (0.5 * (f[i] + f[i + 1]) - WT[i] * rho * (1 + 4.5 * cu * cu - 1.5 * usq)) - gP * WT[i] * (9 * cu * cF - 3 * uF)
            B = om[1] * (0.5 * (f[i] - f[i + 1]) - WT[i] * rho * 3 * cu) - gM * WT[i] * 3 * cF
            post[i] = f[i] - A - B
            post[i + 1] = f[i + 1] - A + B
        for i in range(19):
            f[i] = torch.roll(post[i], (CZ[i], CY[i], CX[i]), (0, 1, 2)) if i else post[0]
        if self.di.numel():
            fp = post.view(19, -1)[self.di, self.ni]
            fb = fp.clone()
            if self.sq and self.part.numel():
                k = self.part
                d, n = self.di[k], self.ni[k]
                c = self.c[d]
                nx, ny = int(self.n[0]), int(self.n[1])
                r = torch.stack([n % nx, (n // nx) % ny, n // (nx * ny)], 1).double() + 0.5 * c - torch.tensor(self.X, device=self.dev)
                for ax in range(3):
                    if not self.wall[ax]:
                        r[:, ax] -= int(self.n[ax]) * torch.round(r[:, ax] / int(self.n[ax]))
                U, W, e = (torch.tensor(v, device=self.dev) for v in (self.U, self.W, self.e))
                rh = r / r.norm(dim=1, keepdim=True)
                ct = (rh @ e).unsqueeze(1)
                ub = U + torch.cross(W.expand_as(r), r, dim=1) + self.p.B1 * (1 + self.p.beta * ct) * (ct * rh - e)
                fb[k] -= 6 * w[d] * rho.reshape(-1)[n] * (c * ub).sum(1)
                dp = (fp[k] + fb[k]).unsqueeze(1) * c - (fp[k] - fb[k]).unsqueeze(1) * ub
                both = torch.cat([dp, torch.cross(r, dp, dim=1)], 1).sum(0).cpu().numpy()
                self.Fh, self.Th = both[:3], both[3:]
            f.view(19, -1)[self.oi, self.ni] = fb

    def advance(self):
        p = self.p
        soft = lambda h: 0.0 if h >= p.hc else p.eps * self.FS * (1 - max(h, 0.0) / p.hc) ** 2  # noqa: E731
        self.Fw = np.zeros(3)
        for d in (1, 2):
            if self.wall[d]:
                self.Fw[d] = soft(self.X[d] - self.R - 0.5) - soft((self.n[d] - 1.5) - self.X[d] - self.R)
        self.U = self.U + (self.Fh + self.Fc + self.Fw) / self.M
        self.W = self.W + (self.Th + self.Tc) / self.I
        self.Fc, self.Tc = np.zeros(3), np.zeros(3)
        if p.planar:
            self.U[2] = self.W[0] = self.W[1] = 0.0
        self.X = self.X + self.U
        self.e = self.e + np.cross(self.W, self.e)
        if p.planar:
            self.e[2] = 0.0
        self.e = self.e / np.linalg.norm(self.e)
        for d in (1, 2):
            if self.wall[d]:
                lo, hi = 0.5 + self.R + p.hmin, (self.n[d] - 1.5) - self.R - p.hmin
                if self.X[d] < lo:
                    self.X[d], self.U[d] = lo, max(self.U[d], 0.0)
                if self.X[d] > hi:
                    self.X[d], self.U[d] = hi, min(self.U[d], 0.0)
        self.remap()

    def remap(self):
        nodes, inside = self.changes(self.flag)
        if not nodes:
            return
        flag = self.flag.copy()
        for (z, y, x), cover in zip(nodes, inside):
            r = self.offset(np.array([x, y, z], float))
            if cover:
                q = C.T @ self.f[:, z, y, x].cpu().numpy()
                self.Fc, self.Tc = self.Fc + q, self.Tc + np.cross(r, q)
                flag[z, y, x] = 2
                continue
            near = [((z + CZ[i]) % self.n[2], (y + CY[i]) % self.n[1], (x + CX[i]) % self.n[0]) for i in range(1, 19)]
            have = [float(self.rho[k]) for k in near if flag[k] == 0]
            rr = sum(have) / len(have) if have else 1.0
            ub = self.U + np.cross(self.W, r)
            cu = C @ ub
            self.f[:, z, y, x] = torch.tensor(WT * rr * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (ub @ ub)), device=self.dev)
            self.rho[z, y, x] = rr
            self.u[z, y, x] = torch.tensor(ub, device=self.dev)
            self.Fc, self.Tc = self.Fc - rr * ub, self.Tc - np.cross(r, rr * ub)
            flag[z, y, x] = 0
        self.set_flag(flag)

    def advance_to(self, steps):
        for k in range(steps):
            self.step(k == steps - 1)
            self.t += 1
            if not self.sq:
                continue
            self.advance()
            if self.t % self.p.massCorrectionEvery == 0:
                d = 1.0 - float((self.f.sum(0) * self.fluid).sum()) / float(self.fluid.sum())
                self.f += self.w.view(19, 1, 1, 1) * d * self.fluid
            if self.t % self.p.trajEvery == 0:
                self.rows.append(np.concatenate([[self.t], self.X, self.e, self.U, self.W, self.Fw[1:]]))

    def squirmer(self):
        return np.stack([self.X, self.e, self.U, self.W, self.Fh, self.Th, self.Fc, self.Tc, self.Fw])


def _exact_net(case, seed):
    """The network's forward, or one epoch of Adam on it, in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    th = torch.tensor(weights(seed), dtype=torch.float64, device=dev)
    x, y = (torch.tensor(v, dtype=torch.float64, device=dev) for v in states(case["n"], seed))
    off = np.cumsum([0, 256, 64, 4096, 64, 4096, 64, 192, 3])
    shapes = [(64, 4), (64,), (64, 64), (64,), (64, 64), (64,), (3, 64), (3,)]

    def parts(v):
        return [v[a:b].view(s) for a, b, s in zip(off[:-1], off[1:], shapes)]

    def layers(v, h):
        q = parts(v)
        zs, hs = [], [h]
        for k in range(0, 6, 2):
            zs.append(hs[-1] @ q[k].T + q[k + 1])
            hs.append(zs[-1] * torch.sigmoid(zs[-1]))
        return q, zs, hs, hs[-1] @ q[6].T + q[7]

    if case["kind"] == "forward":
        return torch.cat([layers(th, h)[3] for h in x.split(1 << 18)])
    order = torch.tensor(np.random.default_rng([19, int(seed)]).permutation(case["n"]), device=dev)
    m, v, losses = torch.zeros_like(th), torch.zeros_like(th), []
    for t, k in enumerate(order.split(case["batch"]), 1):
        q, zs, hs, out = layers(th, x[k])
        d = out - y[k]
        losses.append((d * d).mean())
        d = 2 * d / d.numel()
        g = []
        for j in (3, 2, 1, 0):
            g = [d.T @ hs[j], d.sum(0)] + g
            if j:
                s = torch.sigmoid(zs[j - 1])
                d = (d @ q[2 * j]) * s * (1 + zs[j - 1] * (1 - s))
        g = torch.cat([a.reshape(-1) for a in g])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        th = th - 2e-3 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"loss": float(torch.stack(losses).mean()), "params": th}


def exact(case, seed):
    k = case["kind"]
    if k in ("train", "forward"):
        return _exact_net(case, seed)
    if k in ("lattice", "stepwise"):
        s = Plain64(deck(case, seed), k == "stepwise")
        s.advance_to(case["steps"])
        r = {"flag": None, "rho": s.rho, "u": s.u}
        if s.sq:
            r["squirmer"] = s.squirmer()
            if k == "lattice":
                r["rows"] = np.stack(s.rows) if s.rows else np.zeros((0, 15))
        return r
    ps = members(case, seed)
    if len(ps) * case["steps"] > 800:   # minutes of plain steps
        return None
    done = [Plain64(p, False) for p in ps]
    for s in done:
        s.advance_to(case["steps"])
    r = {"rows": np.concatenate([np.stack(s.rows) for s in done]), "squirmers": np.stack([s.squirmer() for s in done])}
    if case["fields"]:
        r["fields"] = [{"flag": None, "rho": s.rho, "u": s.u} for s in done]
    return r
