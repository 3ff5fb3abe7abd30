"""What the engine is timed on: whole runs of lattice-Boltzmann cases through the public API.

One pass advances a case (or a batch of cases) by a number of time steps and reads the fields back, as a
solver loop does between two outputs; the flow goes on from pass to pass. A step is one call of lbc's
main_lbm. exact() is the same step in FP64 torch, written from lbc's formulas.
"""
import math
import random

import numpy as np
import torch

import lbc_gb300
from lbc_gb300 import cases as lc
from lbc_gb300.abi import dptr

CX, CY, OPP = [0, 1, 0, -1, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1], [0, 3, 4, 1, 2, 7, 8, 5, 6]
WT = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
CS = 1 / math.sqrt(3)
OMEGAS = [0.0, 0.05, 0.1, 0.15, 0.2]  # the impedance wall's tracked frequencies
RING = 4096                           # steps a force history holds
SIZE = {"f64": 8, "f64fma": 8, "f32": 4, "f16": 2}


def listed():
    return [
        # The smallest channel of the smoke test: a step is far shorter than a launch.
        dict(name="channel 64x16 f64", kind="channel", nx=64, ny=16, storage="f64", steps=100),
        # The configured channel (walls, periodic, body force) in lbc's arithmetic.
        dict(name="channel 256x64 f64", kind="channel", nx=256, ny=64, storage="f64", steps=500),
        # A small lid-driven cavity of odd size: Zou-He lid, three walls.
        dict(name="lid 129x129 f32", kind="lid", nx=129, ny=129, storage="f32", steps=1000),
        # lbc's own cylinder (Zou-He inlet, convective outlet, interpolated bounce-back) with the force of
        # every step recorded, at the resolution of its shipped drag record.
        dict(name="cylinder 1000x400 f64", kind="cylinder", nx=1000, ny=400, storage="f64", steps=200),
        # The same case driven as lbc's main does it: main_lbm on the caller's arrays, every step.
        dict(name="main_lbm 1000x400", kind="main_lbm", nx=1000, ny=400, storage="f64", steps=10),
        # Periodic Taylor-Green vortex, FP64: the plain method; and with fused multiply-adds at a ragged size.
        dict(name="vortex 1024x1024 f64", kind="vortex", nx=1024, ny=1024, storage="f64", steps=100),
        dict(name="vortex 1531x1021 fma", kind="vortex", nx=1531, ny=1021, storage="f64fma", steps=150),
        # The large periodic run, FP32-shifted (the headline), and FP16 at an odd size.
        dict(name="vortex 4096x4096 f32", kind="vortex", nx=4096, ny=4096, storage="f32", steps=500),
        dict(name="vortex 3001x2047 f16", kind="vortex", nx=3001, ny=2047, storage="f16", steps=500),
        # Cylinder wake: regularized inlet and outlet, walls, interpolated bounce-back; force of the last step.
        dict(name="wake 2048x512 f32", kind="wake", nx=2048, ny=512, storage="f32", steps=2000),
        # Lid-driven cavity with a moving-wall lid.
        dict(name="cavity 2048x2048 f32", kind="cavity", nx=2048, ny=2048, storage="f32", steps=500),
        # 64 liner ducts of uneven size with impedance walls in one batch (a sweep).
        dict(name="64 ducts f32", kind="ducts", nx=2048, ny=256, count=64, storage="f32", steps=500, mix=2026),
    ]


def draw(rng):
    """Sizes over the listed ranges, odd ones among them; steps keep a pass within the largest listed one."""
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["channel", "lid", "cylinder", "main_lbm", "vortex", "vortex", "wake", "cavity", "ducts"])
    storage = "f64" if kind == "main_lbm" else "f32" if kind == "ducts" else rng.choice(["f64", "f64fma", "f32", "f32", "f16"])
    if kind == "ducts":
        return dict(kind=kind, nx=log(256, 2048), ny=log(48, 256), count=rng.randint(3, 64), storage=storage,
                    steps=rng.randint(100, 500), mix=rng.randrange(1 << 20))
    if kind in ("cylinder", "main_lbm"):
        ny = log(80, 800)
        nx = 5 * ny // 2
    elif kind == "wake":
        ny = log(64, 768)
        nx = 4 * ny + rng.randint(-7, 7)
    elif kind in ("lid", "cavity"):
        nx = ny = log(64, 2048)
    else:
        nx, ny = log(64, 4096), log(16, 2500)
    if storage == "f16" and kind != "vortex":  # FP16 storage is for periodic and qualitative runs
        storage = "f32"
    most = 3e8 if storage.startswith("f64") else 4e9
    steps = 10 if kind == "main_lbm" else max(20, min(log(100, 1000), int(most / (nx * ny))))
    return dict(kind=kind, nx=nx, ny=ny, storage=storage, steps=steps)


# ---------------------------------------------------------------- geometry and initial fields

def _modes(rng, nx, ny, amp):
    """A seeded smooth field, a few waves of the box, on the GPU."""
    x = torch.arange(nx, dtype=torch.float64, device="cuda")[None, :] * (2 * math.pi / nx)
    y = torch.arange(ny, dtype=torch.float64, device="cuda")[:, None] * (2 * math.pi / ny)
    f = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
    for _ in range(4):
        f += amp * rng.uniform(-1, 1) * torch.sin(rng.randint(1, 3) * x + rng.uniform(0, 6.28)) * torch.cos(rng.randint(1, 3) * y + rng.uniform(0, 6.28))
    return f


def _geometry(kind, nx, ny, **p):
    """Walls, relaxation, boundary list (name, line, val1, val2) and mean flow of one case."""
    mask = np.zeros((ny, nx), np.int32)
    g = dict(kind=kind, nx=nx, ny=ny, mask=mask, phi=np.zeros((ny, nx)), bcs=[], F=0.0, ibb=0, wall_u=None, tau=0.6, u=np.zeros((ny, nx)), imp=None)
    y = np.arange(ny) - 0.5
    if kind == "channel":
        mask[0] = mask[-1] = 1
        g.update(bcs=[("periodic_x", 0, None, None)], F=1e-6, tau=0.8)
    elif kind == "vortex":
        g.update(bcs=[("periodic_x", 0, None, None), ("periodic_y", 0, None, None)], tau=0.56)
        kx, ky = 2 * math.pi / nx, 2 * math.pi / ny
        g.update(u=None, wave=(kx, ky))
    elif kind in ("lid", "cavity"):
        mask[0] = mask[:, 0] = mask[:, -1] = 1
        g["tau"] = 0.5 + 3 * 0.1 * (nx - 2) / (max(100.0, nx) if kind == "lid" else 1000.0)
        if kind == "lid":
            g["bcs"] = [("velocity_top", ny - 1, np.full(nx, 0.1), np.zeros(nx))]
        else:
            mask[-1] = 1
            g["wall_u"] = np.zeros((ny, nx))
            g["wall_u"][-1, 1:-1] = 0.1
    elif kind in ("cylinder", "main_lbm"):
        d = np.sqrt((np.arange(nx)[None, :] - nx / 4) ** 2 + (np.arange(ny)[:, None] - ny / 2) ** 2)
        R, U = ny / 20, 0.05
        mask[d <= R] = 1
        g.update(phi=d - R, ibb=1, tau=0.5 + 3 * U * 2 * R / 20.0, u=np.full((ny, nx), U),
                 bcs=[("periodic_y", 0, None, None), ("velocity_inlet", 0, np.full(ny, U), np.zeros(ny)),
                      ("convective_outlet", nx - 1, np.ones(ny), np.zeros(ny))])
    elif kind == "wake":
        d = np.sqrt((np.arange(nx)[None, :] - nx / 4) ** 2 + (np.arange(ny)[:, None] - ny / 2) ** 2)
        R, U = ny / 16, 0.05
        mask[d <= R] = 1
        mask[0] = mask[-1] = 1
        prof = 4 * U * y * (ny - 2 - y) / (ny - 2) ** 2
        prof[0] = prof[-1] = 0
        g.update(phi=d - R, ibb=1, tau=0.5 + 3 * U * 2 * R / 100.0, u=np.repeat(prof[:, None], nx, 1),
                 bcs=[("velocity_inlet_regularized", 0, prof, np.zeros(ny)), ("pressure_outlet_regularized", nx - 1, np.ones(ny), np.zeros(ny))])
    else:  # duct: grazing flow over a liner in the middle of the bottom row
        u0 = p["mach"] * CS
        i0, i1 = int(round(nx * 0.3)), int(round(nx * 0.7))
        mask[0] = mask[-1] = 1
        mask[0, i0:i1] = 0
        R, m, K = np.zeros(nx), np.zeros(nx), np.zeros(nx)
        R[i0:i1], m[i0:i1], K[i0:i1] = p["R"], p["m"], p["m"] * (2 * math.pi * p["f"]) ** 2
        g.update(u=np.full((ny, nx), u0), imp=(2, R, m, K, 1e-3, 20000),
                 bcs=[("velocity_inlet_regularized", 0, np.full(ny, u0), np.zeros(ny)), ("pressure_outlet_regularized", nx - 1, np.ones(ny), np.zeros(ny)),
                      ("velocity_bottom_regularized", 0, np.zeros(nx), np.zeros(nx))])
    return g


def _cases(case):
    if case["kind"] != "ducts":
        return [_geometry(case["kind"], case["nx"], case["ny"])]
    r = random.Random(case["mix"])
    return [_geometry("duct", r.randint(max(64, case["nx"] // 4), case["nx"]), r.randint(max(24, case["ny"] // 4), case["ny"]), mach=r.uniform(0, 0.3),
                      R=r.uniform(0.5, 3) * CS, m=r.uniform(1e-3, 1e-2), f=r.uniform(0.02, 0.1)) for _ in range(case["count"])]


def _fields(g, seed):
    """Seeded initial rho, u, v of one case, FP64 on the GPU."""
    rng = random.Random(seed)
    nx, ny = g["nx"], g["ny"]
    fluid = torch.from_numpy(1.0 - g["mask"]).cuda()
    rho = 1 + _modes(rng, nx, ny, 1e-3 if g["imp"] else 1e-4) * fluid
    if g["u"] is None:
        kx, ky = g["wave"]
        x = torch.arange(nx, dtype=torch.float64, device="cuda")[None, :] * kx + rng.uniform(0, 6.28)
        y = torch.arange(ny, dtype=torch.float64, device="cuda")[:, None] * ky + rng.uniform(0, 6.28)
        a = 0.04 / math.sqrt(max(kx / ky, ky / kx))
        return rho, -a * math.sqrt(ky / kx) * torch.cos(x) * torch.sin(y) + _modes(rng, nx, ny, 1e-3), a * math.sqrt(kx / ky) * torch.sin(x) * torch.cos(y)
    u = torch.from_numpy(g["u"]).cuda() * fluid
    return rho, u + _modes(rng, nx, ny, 2e-3) * fluid, _modes(rng, nx, ny, 2e-3) * fluid


def _equilibrium(rho, u, v):
    f = torch.empty(rho.shape + (9,), dtype=torch.float64, device="cuda")
    for k in range(9):
        cu = CX[k] * u + CY[k] * v
        f[..., k] = WT[k] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (u * u + v * v))
    return f


# ---------------------------------------------------------------- a pass

_tables = {}


def _case(key, g):
    """The Case of one geometry: main_lbm callers keep their tables from run to run, so its states share them."""
    if key not in _tables:
        ny, nx = g["ny"], g["nx"]
        made = lc.Case(g["kind"], nx, ny, g["mask"], np.full((ny, nx), 1 / g["tau"]), g["phi"], [lc.BC(*b) for b in g["bcs"]], Fx=g["F"],
                       use_IBB=g["ibb"], wall_u=g["wall_u"])
        if g["kind"] != "main_lbm":
            return made
        _tables.clear()
        _tables[key] = made
    return _tables[key]


def prepare(case, seed):
    sims = []
    for n, g in enumerate(_cases(case)):
        c = _case(str(sorted(case.items())), g)
        rho, u, v = _fields(g, 1000 * seed + n)
        f = _equilibrium(rho, u, v).cpu().numpy()
        st = lc.State(f, f.copy() if case["kind"] == "main_lbm" else f, rho.cpu().numpy(), u.cpu().numpy(), v.cpu().numpy())
        if case["kind"] == "main_lbm":
            api = lbc_gb300.dropin()
            return dict(case=case, api=api, c=c, st=st, bnd=api.boundaries(c.bcs))
        s = lbc_gb300.GpuSolver(c, lbc_gb300.STORAGE[case["storage"]])
        if g["imp"]:
            entry, R, m, K, alpha, window = g["imp"]
            s.set_impedance_wall(entry, R, m, K, OMEGAS, 1.0, alpha, window)
        if case["kind"] == "cylinder":
            s.enable_force_history(RING)
        s.set_state(st)
        sims.append((s, c))
    # one results array a quantity, kept from output to output
    at = np.cumsum([0] + [c.nodes for _, c in sims])
    out = [np.zeros(at[-1]) for _ in range(3)]
    into = [[dptr(o[a:]) for o in out] for a in at[:-1]]
    batch = lbc_gb300.GpuBatch([s for s, _ in sims]) if case["kind"] == "ducts" else None
    return dict(case=case, sims=sims, batch=batch, out=out, into=into)


def run(state):
    case = state["case"]
    if case["kind"] == "main_lbm":
        api, c, st = state["api"], state["c"], state["st"]
        force = [api.step(c, st, state["bnd"]) for _ in range(case["steps"])]
        return dict(f=st.f, f_new=st.f_new, rho=st.rho, u=st.u, v=st.v, force=np.array(force))
    (state["batch"] or state["sims"][0][0]).run(case["steps"])
    for (s, _), ptr in zip(state["sims"], state["into"]):
        if s.lib.lbm_gpu_get_fields(s.h, *ptr) != 0:
            raise RuntimeError(lbc_gb300.last_error())
    got = dict(zip(("rho", "u", "v"), state["out"]))
    s = state["sims"][0][0]
    if case["kind"] == "cylinder":
        got["force"] = s.force_history(RING)[-case["steps"]:]
    elif case["kind"] in ("channel", "wake", "cavity"):
        got["force"] = np.array(s.forces())
    elif case["kind"] == "ducts":
        got["spectra"] = np.concatenate([d.impedance_readback(2)[0] for d, _ in state["sims"]])
    return got


def work(case):
    """Each state read once and written once, in its storage type, and the fields; the step's arithmetic (lbc's expression count)."""
    n = sum(g["nx"] * g["ny"] for g in _cases(case))
    size = SIZE[case["storage"]]
    return {"bytes": n * (2 * 9 * size + 24), "flops": 150.0 * n * case["steps"]}


# ---------------------------------------------------------------- the same in 64 bits

class _Exact:
    """lbc's step on [9, Ny, Nx] FP64 tensors, captured once and replayed."""

    def __init__(self, g, seed):
        T = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        self.g, nx, ny = g, g["nx"], g["ny"]
        names = [b[0] for b in g["bcs"]]
        px, py = "periodic_x" in names, "periodic_y" in names
        self.rho, self.u, self.v = (t.clone() for t in _fields(g, seed))
        self.f = _equilibrium(self.rho, self.u, self.v).permute(2, 0, 1).contiguous()
        self.fn = self.f.clone()
        self.c = [T(a)[:, None, None] for a in (CX, CY, WT)]
        solid = torch.from_numpy(g["mask"].astype(bool)).cuda()
        self.solid, n = solid, nx * ny
        self.nan = torch.where(solid, math.nan, 0.0).to(torch.float64)
        node = torch.arange(n, device="cuda").view(ny, nx)
        x, y = node % nx, node // nx

        def at(dx, dy):
            """(linear node at +dx, +dy; whether it is on the grid)"""
            i, j = x + dx, y + dy
            on = torch.ones_like(solid)
            on &= torch.ones_like(solid) if px else (i >= 0) & (i < nx)
            on &= torch.ones_like(solid) if py else (j >= 0) & (j < ny)
            return (j % ny) * nx + i % nx, on

        src, keep, lk = [], [], {a: [] for a in ("to", "own", "behind", "c1", "c2", "add", "cx", "cy")}
        phi, uw = T(g["phi"]).view(-1), T(g["wall_u"] if g["wall_u"] is not None else np.zeros((ny, nx))).view(-1)
        for k in range(9):
            s, on = at(-CX[k], -CY[k])
            hit = solid.view(-1)[s] & on & ~solid
            src.append(torch.where(hit, OPP[k] * n + node, k * n + s))
            keep.append(solid | ~on)
            if k and bool(hit.any()):  # links into the wall along opp k, reflected into k
                own = node[hit]
                wall = s[hit]
                b, bon = (t[hit] for t in at(CX[k], CY[k]))
                one = torch.ones(len(own), dtype=torch.float64, device="cuda")
                c1, c2, behind = one.clone(), 0 * one, own + OPP[k] * n
                if g["ibb"]:
                    den = phi[own] - phi[wall]
                    den = torch.where(den.abs() < 1e-12, torch.where(den >= 0, 1e-12, -1e-12).to(den), den)
                    q = (phi[own] / den).clamp(1e-12, 1 - 1e-12)
                    lo, hi = bon & (q <= 0.5), bon & (q > 0.5) & ~solid.view(-1)[b]
                    c1 = torch.where(lo, 1 - 2 * q, torch.where(hi, 1 / (2 * q), one))
                    c2 = torch.where(lo, 2 * q, torch.where(hi, (2 * q - 1) / (2 * q), 0 * one))
                    behind = torch.where(lo, b + OPP[k] * n, torch.where(hi, b + k * n, behind))
                for name, val in (("to", own + k * n), ("own", own + OPP[k] * n), ("behind", behind), ("c1", c1), ("c2", c2),
                                  ("add", -6 * WT[k] * CX[OPP[k]] * uw[wall]), ("cx", -CX[k] * one), ("cy", -CY[k] * one)):
                    lk[name].append(val)
        self.src, self.keep = torch.stack(src), torch.stack(keep)
        self.links = {a: torch.cat(v) for a, v in lk.items()} if lk["to"] else None
        self.force = torch.zeros(2, dtype=torch.float64, device="cuda")
        self.bcs = [(b[0], b[1], None if b[2] is None else T(b[2]), None if b[3] is None else T(b[3])) for b in g["bcs"]]
        if g["imp"]:
            _, R, m, K, self.alpha, window = g["imp"]
            on = np.flatnonzero(m)
            M = T(np.array([[[0, 1], [-K[t] / m[t], -R[t] / m[t]]] for t in on[:1]]))
            A = torch.linalg.matrix_exp(M)[0]
            b = torch.linalg.solve(M[0], (A - torch.eye(2).to(A)) @ T([0.0, 1 / m[on[0]]]))
            self.on, self.A, self.b = torch.from_numpy(on).cuda(), A, b
            self.rb, self.xv = torch.ones(len(on)).to(A), torch.zeros(2, len(on)).to(A)
            self.spec = torch.zeros(g["nx"], len(OMEGAS), 4).to(A)
            self.turn = torch.tensor([2 * math.pi / window] + [-w for w in OMEGAS], dtype=torch.float64, device="cuda")
            self.angle = torch.zeros_like(self.turn)

    def _feq(self, rho, u, v, c):
        cu = c[0] * u + c[1] * v
        return c[2] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (u * u + v * v))

    def _line(self, name, at):
        """Edge line and its interior neighbour as index tuples."""
        if "inlet" in name or "outlet" in name:
            return (slice(None), at), (slice(None), at + (1 if "inlet" in name else -1))
        return (at, slice(None)), (at + (1 if "bottom" in name else -1), slice(None))

    def step(self):
        f, c, g = self.f, self.c, self.g
        om, F = 1 / g["tau"], g["F"]
        fc = f - om * (f - self._feq(self.rho, self.u, self.v, c))
        if F:
            cu = c[0] * self.u + c[1] * self.v
            fc = fc + (1 - 0.5 * om) * c[2] * (3 * c[0] * F + 9 * cu * c[0] * F - 3 * self.u * F)
        fc = torch.where(self.solid, f, fc)
        new = torch.where(self.keep, self.fn, fc.view(-1)[self.src])
        if self.links:
            k = self.links
            flat, own = new.view(-1), fc.view(-1)[k["own"]]
            back = k["c1"] * own + k["c2"] * fc.view(-1)[k["behind"]] + k["add"]
            flat[k["to"]] = back
            self.force.copy_(torch.stack([((own + back) * k["cy"]).sum(), ((own + back) * k["cx"]).sum()]))  # L, D
        for name, at, a, b in self.bcs:
            if name.startswith("periodic"):
                continue
            e, i = self._line(name, at)
            E, I = (slice(None),) + e, (slice(None),) + i
            p, ok = new[E].clone(), ~self.solid[e]
            if name == "convective_outlet":
                q = new[I]
            elif name == "velocity_inlet":
                r = (p[0] + p[2] + p[4] + 2 * (p[3] + p[6] + p[7])) / (1 - a)
                d = 0.5 * (p[2] - p[4])
                q = torch.stack([p[0], p[3] + 2 / 3 * r * a, p[2], p[3], p[4], p[7] + r * a / 6 - d + r * b / 2, p[6], p[7], p[6] + r * a / 6 + d - r * b / 2])
            elif name == "velocity_top":
                r = (p[0] + p[1] + p[3] + 2 * (p[2] + p[5] + p[6])) / (1 + b)
                d = 0.5 * (p[1] - p[3])
                q = torch.stack([p[0], p[1], p[2], p[3], p[2] - 2 / 3 * r * b, p[5], p[6], p[5] + d - r * a / 2 - r * b / 6, p[6] - d + r * a / 2 - r * b / 6])
            else:
                c1 = [t[:, :, 0] for t in c]
                rn, un, vn = self.rho[i], self.u[i], self.v[i]
                if g["imp"] and "bottom" in name:
                    b = self._wall(rn, b)
                rb, ub, vb = (a, un, vn) if "pressure" in name else (rn, a, b)
                ne = new[I] - self._feq(rn, un, vn, c1)
                xx, yy = c1[0] * c1[0], c1[1] * c1[1]
                Pxx, Pxy, Pyy = (xx * ne).sum(0), (c1[0] * c1[1] * ne).sum(0), (yy * ne).sum(0)
                q = self._feq(rb, ub, vb, c1) + 1.5 * c1[2] * ((xx - 1 / 3) * Pxx + 2 * c1[0] * c1[1] * Pxy + (yy - 1 / 3) * Pyy)
            new[E] = torch.where(ok, q, p)
        rho = new.sum(0)
        self.u.copy_(((new * c[0]).sum(0) + F / 2) / rho + self.nan)
        self.v.copy_((new * c[1]).sum(0) / rho + self.nan)
        self.rho.copy_(rho + self.nan)
        self.fn.copy_(fc)
        self.f.copy_(new)

    def _wall(self, rn, given):
        p = (rn[self.on] - self.rb) / 3
        self.rb.add_(self.alpha * 3 * p)
        self.xv.copy_(self.A @ self.xv + self.b[:, None] * p)
        win = 0.5 * (1 - torch.cos(self.angle[0]))
        c, s = torch.cos(self.angle[1:]), torch.sin(self.angle[1:])
        P, V = win * p[:, None], win * self.xv[1][:, None]
        self.spec.index_add_(0, self.on, torch.stack([P * c, P * s, V * c, V * s], -1))
        self.angle.add_(self.turn)
        return given.index_copy(0, self.on, -self.xv[1])

    def go(self, steps, record):
        got = []
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            self.step()
            got.append(self.force.clone())
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            self.step()
        for _ in range(steps - 1):
            graph.replay()
            if record:
                got.append(self.force.clone())
        return torch.stack(got) if record else self.force


def exact(case, seed):
    sims = []
    for n, g in enumerate(_cases(case)):
        e = _Exact(g, 1000 * seed + n)
        force = e.go(case["steps"], case["kind"] in ("cylinder", "main_lbm"))
        sims.append((e, force))
    e, force = sims[0]
    if case["kind"] == "main_lbm":
        return dict(f=e.f.permute(1, 2, 0), f_new=e.fn.permute(1, 2, 0), rho=e.rho, u=e.u, v=e.v, force=force)
    got = {k: torch.cat([getattr(s, k).reshape(-1) for s, _ in sims]) for k in ("rho", "u", "v")}
    if case["kind"] == "cylinder":
        got["force"] = force.flip(1)
    elif case["kind"] in ("channel", "wake", "cavity"):
        got["force"] = force
    elif case["kind"] == "ducts":
        got["spectra"] = torch.cat([s.spec for s, _ in sims])
    return got
