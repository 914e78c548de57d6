"""Performance cases of the rans residual path.

Each case is work that a program does through the public interface
(aeroflex_gb300.rans): residual evaluations, explicit and implicit
iterations, batches of load cases and the vector-Jacobian product of the
adjoint, from a thousand cells to four million, FP64 and FP32-mixed.  The
meshes are those of the tests and the benchmark (aeroflex_gb300.meshgen) and
odd sizes of the same generators.

An FP64 solver's fields are returned in FP64.  An FP32-mixed solver's fields
are handed on in FP32, the precision that path computes in, as a viewer or a
learning pipeline takes them.
"""
import functools
import math

import numpy as np
import torch

from aeroflex_gb300 import meshgen, rans

DEG = 0.01745  # the reference's degree -> radian factor
GAMMA, RGAS, PR_L, RELAX, LIM_K = 1.4, 0.71428571428, 0.72, 0.9, 5.0


def _case(name, do, mesh, **kw):
    c = dict(name=name, do=do, mesh=mesh, a=0, b=0, split=False, precision="fp64", solver="explicit",
             viscosity="inviscid", wall="slip-wall", gradient="green-gauss", limiter="venkatakrishnan", second=True,
             cfl=1.0, mu=1e-5, mach=0.5, aoa=1.25, steps=1, cases=0, fill=0)
    for k in kw:
        if k not in c:
            raise KeyError(k)
    c.update(kw)
    return c


def listed():
    return [
        # one residual of a coarse test mesh from a host state: the smallest call a coupling or a
        # unit test makes, all latency
        _case("residual_1k_f64", "residual", "omesh", a=32, b=16, split=True),
        # the bit-exact explicit solver on the classic 128 x 64 O-mesh split into triangles, with the
        # wall forces read after it: a polar point in progress
        _case("explicit_16k_f64", "explicit", "omesh", a=128, b=64, split=True, steps=50),
        # a viscous run with the other options (no-slip wall, least squares, Michalak) on an odd mesh,
        # in FP32-mixed: how a user iterates quickly on a small case
        _case("laminar_17k_f32", "explicit", "omesh", a=201, b=83, precision="fp32-mixed", viscosity="laminar",
              wall="wall", gradient="least-squares", limiter="michalak", mu=2e-4, mach=0.3, aoa=2.0, steps=50),
        # the laminar FP64 path at a medium size (quadrilaterals)
        _case("laminar_74k_f64", "explicit", "omesh", a=384, b=192, viscosity="laminar", wall="wall", mu=2e-4,
              mach=0.3, aoa=2.0, steps=6),
        # a large FP64 flow field, the precision the reference computes in
        _case("channel_1m_f64", "explicit", "channel", a=1024, b=512, mach=0.3, aoa=0.0, steps=3),
        # the throughput configuration: 4.19M shuffled triangles, FP32-mixed
        _case("channel_4m_f32", "explicit", "channel", a=2048, b=1024, precision="fp32-mixed", mach=0.3, aoa=0.0,
              steps=10),
        # the reference's default solver, implicit, on the 128 x 128 airfoil in FP64
        _case("implicit_16k_f64", "implicit", "omesh", a=128, b=128, solver="implicit", cfl=40.0, steps=2),
        # the same solver in FP32-mixed on a fine airfoil
        _case("implicit_131k_f32", "implicit", "omesh", a=512, b=256, precision="fp32-mixed", solver="implicit",
              cfl=40.0, steps=1),
        # a RANS run: Spalart-Allmaras, Re 6e6, hybrid boundary-layer mesh (201k cells), first order
        _case("sa_201k_f32", "implicit", "hybrid", a=512, b=60, fill=170000, precision="fp32-mixed",
              solver="implicit", viscosity="spalart-allmaras", wall="wall", second=False, mu=1.4 * 0.15 / 6e6,
              mach=0.15, aoa=10.0, cfl=20.0, steps=1),
        # a polar sweep's load cases advanced together, explicit, FP32-mixed
        _case("sweep24_f32", "batch", "sweep", a=5000, b=60000, precision="fp32-mixed", cases=24, steps=20),
        # load cases advanced together by the implicit solver
        _case("sweep8_implicit_f32", "batch", "sweep", a=5000, b=40000, precision="fp32-mixed", solver="implicit",
              cfl=40.0, cases=8, steps=1),
        # the adjoint's vector-Jacobian product on a quarter of a million cells
        _case("vjp_262k_f64", "vjp", "channel", a=512, b=256, mach=0.3, aoa=0.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds: sizes spread over their logarithm, odd ones among them."""
    c = _draw(rng)
    del c["name"]
    return c


def _draw(rng):
    kind = rng.choice(["residual", "explicit", "explicit", "laminar", "channel", "implicit", "sa", "sweep",
                       "sweep_implicit", "vjp"])
    prec = rng.choice(["fp64", "fp32-mixed"])
    mach, aoa = round(rng.uniform(0.2, 0.6), 3), round(rng.uniform(-2.0, 5.0), 2)
    if kind == "residual":
        nr = _log(rng, 8, 120)
        return _case("", "residual", "omesh", a=2 * nr + rng.randrange(3), b=nr, split=rng.random() < 0.5,
                     precision=prec, mach=mach, aoa=aoa, limiter=rng.choice(["venkatakrishnan", "michalak"]))
    if kind == "explicit":
        nr = _log(rng, 20, 300)
        return _case("", "explicit", "omesh", a=2 * nr + rng.randrange(3), b=nr, split=rng.random() < 0.5,
                     precision=prec, mach=mach, aoa=aoa, second=rng.random() < 0.8,
                     gradient=rng.choice(["green-gauss", "green-gauss", "least-squares"]),
                     steps=max(2, 400 // nr))
    if kind == "laminar":
        nr = _log(rng, 20, 220)
        return _case("", "explicit", "omesh", a=2 * nr + rng.randrange(3), b=nr, split=rng.random() < 0.5,
                     precision=prec, viscosity="laminar", wall="wall", mu=2e-4, mach=round(rng.uniform(0.2, 0.4), 3),
                     aoa=aoa, limiter=rng.choice(["venkatakrishnan", "michalak"]), steps=max(2, 300 // nr))
    if kind == "channel":
        ny = _log(rng, 64, 1000 if prec == "fp32-mixed" else 500)
        return _case("", "explicit", "channel", a=2 * ny + rng.randrange(3), b=ny, precision=prec, mach=mach, aoa=0.0,
                     steps=3 if prec == "fp64" else 10)
    if kind == "implicit":
        nr = _log(rng, 24, 256 if prec == "fp32-mixed" else 160)
        return _case("", "implicit", "omesh", a=2 * nr + rng.randrange(3), b=nr, precision=prec, solver="implicit",
                     mach=mach, aoa=aoa, cfl=40.0, steps=1)
    if kind == "sa":
        ns = _log(rng, 128, 450)
        return _case("", "implicit", "hybrid", a=ns, b=60, fill=int(170000 * (ns / 512.0) ** 2),
                     precision=prec if ns < 300 else "fp32-mixed", solver="implicit", viscosity="spalart-allmaras",
                     wall="wall", second=False, mu=1.4 * 0.15 / 6e6, mach=0.15, aoa=round(rng.uniform(0.0, 10.0), 2),
                     cfl=20.0, steps=1)
    if kind == "sweep":
        n = rng.randrange(3, 25)
        prec = "fp32-mixed" if n > 8 else prec
        return _case("", "batch", "sweep", a=_log(rng, 1500, 5000), b=_log(rng, 8000, 60000), precision=prec, cases=n,
                     steps=20 if prec == "fp32-mixed" else 4)
    if kind == "sweep_implicit":
        return _case("", "batch", "sweep", a=_log(rng, 1500, 5000), b=_log(rng, 8000, 40000), precision="fp32-mixed",
                     solver="implicit", cfl=40.0, cases=rng.randrange(2, 9), steps=1)
    ny = _log(rng, 32, 256)
    return _case("", "vjp", "channel", a=2 * ny + rng.randrange(3), b=ny, mach=mach, aoa=0.0,
                 viscosity=rng.choice(["inviscid", "laminar"]), mu=2e-4, second=rng.random() < 0.7)


# ------------------------------------------------------------------ meshes
@functools.lru_cache(maxsize=6)
def _arrays(kind, a, b, split, fill):
    if kind == "channel":
        return meshgen.channel(a, b)
    if kind == "hybrid":
        # the generator refuses a fill whose last ring crowds the far-field circle: the next size then
        for k in range(40):
            try:
                return meshgen.hybrid_airfoil(n_surf=a, bl_layers=b, fill_cells=int(fill * (1.0 + 0.013 * k)))
            except RuntimeError:
                if k == 39:
                    raise
    return meshgen.airfoil_omesh(n_surf=a, n_rad=b, split=split, fade=2 if b > 150 else 1)


@functools.lru_cache(maxsize=2)
def _sweep(n, lo, hi):
    return meshgen.polar_sweep_cases(n, n_min=lo, n_max=hi)


@functools.lru_cache(maxsize=4)
def _mesh(kind, a, b, split, fill):
    """The mesh a program has loaded, and its cell centroids."""
    m = _arrays(kind, a, b, split, fill)
    cx, cy = meshgen.cell_centroids(m)
    return rans.mesh.from_arrays(m), torch.from_numpy(cx), torch.from_numpy(cy)


@functools.lru_cache(maxsize=2)
def _sweep_meshes(n, lo, hi):
    out = []
    for c in _sweep(n, lo, hi):
        cx, cy = meshgen.cell_centroids(c["mesh"])
        out.append((rans.mesh.from_arrays(c["mesh"]), torch.from_numpy(cx), torch.from_numpy(cy)))
    return out


def _freestream(mach, angle):
    rho = 1.0 / RGAS
    c = math.sqrt(GAMMA * RGAS)
    u, v = mach * c * math.cos(angle), mach * c * math.sin(angle)
    return rho, u, v


def _flow(cx, cy, mach, angle, seed):
    """A smooth disturbed stream around the body: freestream with a few waves of 1-2 % in density,
    velocity and pressure, [rho, rhou, rhov, rhoE] per cell, flat FP64."""
    rho, u, v = _freestream(mach, angle)
    r = np.random.default_rng(seed)
    x, y = torch.atan(cx - 0.5), torch.atan(cy - 0.5)  # waves near the body, none far away
    w = []
    for amp in (0.02, 0.01, 0.01, 0.015):
        k1, k2, ph = r.uniform(2.0, 9.0), r.uniform(2.0, 9.0), r.uniform(0.0, 2 * math.pi)
        w.append(amp * torch.sin(k1 * x + k2 * y + ph))
    rho = rho * (1.0 + w[0])
    u, v, p = u + 0.5 * w[1], v + 0.5 * w[2], 1.0 + w[3]
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], 1).reshape(-1)


def _settings(c, mach, angle):
    s = rans.Settings().set("solver", c["solver"]).set("precision", c["precision"])
    s.set("viscosity", c["viscosity"]).set("gradient", c["gradient"]).set("limiter", c["limiter"])
    s.set("second_order", 1.0 if c["second"] else 0.0).set("mu_L", c["mu"]).set("relaxation", RELAX)
    s.set("limiter_k", LIM_K).set("start_cfl", c["cfl"])
    if c["solver"] == "implicit":
        s.set("max_cfl", max(100.0, c["cfl"]))
    s.set_bc("farfield", "farfield", 1.0, mach, angle, 1.0).set_bc("wall", c["wall"])
    return s


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available())


# ------------------------------------------------------------------ states
def prepare(case, seed):
    c = dict(case)
    if c["do"] == "batch":
        flow = _sweep(c["cases"], c["a"], c["b"])
        meshes = _sweep_meshes(c["cases"], c["a"], c["b"])
        batch = rans.Batch([m for m, _, _ in meshes], [_settings(c, f["mach"], f["aoa_deg"] * DEG) for f in flow])
        q = [_flow(cx, cy, f["mach"], f["aoa_deg"] * DEG, seed * 1000 + k).numpy()
             for k, ((_, cx, cy), f) in enumerate(zip(meshes, flow))]
        return dict(case=c, batch=batch, q=q)
    m, cx, cy = _mesh(c["mesh"], c["a"], c["b"], c["split"], c["fill"])
    s = rans.Solver(m, _settings(c, c["mach"], c["aoa"] * DEG))
    s.init()
    q = _pinned(4 * m.nRealCells)
    q.copy_(_flow(cx, cy, c["mach"], c["aoa"] * DEG, seed))
    st = dict(case=c, solver=s, q=q.numpy(), keep=q)
    if c["do"] == "vjp":
        g = torch.Generator().manual_seed(seed)
        st["v"] = torch.randn(4 * m.nRealCells, generator=g, dtype=torch.float64).numpy()
    else:
        out = _pinned(4 * m.nRealCells)
        st["out"], st["keep_out"] = out.numpy(), out
    return st


def _handed_on(x, c):
    t = torch.from_numpy(x)
    return t if c["precision"] == "fp64" else t.float()


def run(state):
    c = state["case"]
    if c["do"] == "batch":
        b = state["batch"]
        for k in range(len(b)):
            b.set_q(k, state["q"][k])
        b.iterate(c["steps"])
        return [_handed_on(b.get_q(k), c) for k in range(len(b))]
    s = state["solver"]
    if c["do"] == "vjp":
        u, bq = s.residual_vjp(state["v"], q=state["q"])
        return dict(u=u, bq=bq)
    s.set_q(state["q"])
    if c["do"] == "residual":
        return dict(R=_handed_on(s.residual(), c))
    if c["viscosity"] == "spalart-allmaras":
        s.set_nu(np.full(s.n_real, 3.0 * c["mu"] * RGAS))
    s.iterate(c["steps"])
    out = dict(q=_handed_on(s.get_q(state["out"]), c))
    if c["viscosity"] == "spalart-allmaras":
        out["nu"] = _handed_on(s.nu(), c)
    if c["mesh"] != "channel":
        w = rans.get_wall_profile(s, "wall", cap=4096)
        f = float if c["precision"] == "fp64" else np.float32
        out.update(cl=f(w["cl"]), cd=f(w["cd"]), cm=f(w["cm"]), cp=_handed_on(w["cp"], c))
    return out


# ------------------------------------------------------------------ work
def _counts(c):
    """(cells, faces, boundary faces) without making the mesh."""
    if c["mesh"] == "channel":
        a, b = c["a"], c["b"]
        return 2 * a * b, 3 * a * b + a + b, 2 * (a + b)
    if c["mesh"] == "hybrid":
        n = c["a"] * c["b"] + c["fill"]
        return n, 2 * c["a"] * c["b"] + 3 * c["fill"] // 2, c["a"] + 128
    if c["mesh"] == "sweep":
        # log-uniform sizes: their mean
        n = int(c["cases"] * (c["b"] - c["a"]) / max(1e-9, math.log(c["b"] / c["a"])))
        return n, 2 * n, int(math.sqrt(8.0 * n * c["cases"]))
    n = c["a"] * c["b"]
    return (2 * n, 3 * n + c["a"], 2 * c["a"]) if c["split"] else (n, 2 * n + c["a"], 2 * c["a"])


def work(case):
    """Bytes: every array of an evaluation once (states and ghosts, geometry, gradients and limiter written and
    read, result), per evaluation.  Operations: the scheme's, hand-counted (face flux 207, reconstruction 44,
    limiter 230, sums 12 per face and evaluation; gradient and time step 111 per face and iteration)."""
    c = case
    n, f, g = _counts(c)
    w = 8 if c["precision"] == "fp64" else 4
    ev = (n + g) * 7 * w + n * (24 * w * (1 if c["second"] else 0) + 32) + f * (8 + 5 * w)
    visc = 0 if c["viscosity"] == "inviscid" else 150
    ops = f * (219 + visc + (274 if c["second"] else 0))
    per_it = f * 111 + n * 70
    if c["do"] == "residual":
        return {"bytes": ev + 64 * n, "flops": ops + f * 73}
    if c["do"] == "vjp":
        # states, weights and result; about four evaluations' arithmetic
        return {"bytes": ev + 96 * n, "flops": 4 * ops}
    if c["solver"] == "implicit":
        # fill, right-hand sides and at least six Krylov steps of the block system per iteration
        blocks = n * (16 + 64) * w
        it = 7 * ev + blocks + 6 * (2 * blocks + 20 * n * w)
        return {"bytes": c["steps"] * it + 64 * n, "flops": c["steps"] * (7 * ops + 9 * f * (207 + visc) + 6 * n * 320)}
    return {"bytes": c["steps"] * 3 * ev + 64 * n, "flops": c["steps"] * (3 * ops + per_it)}


# ------------------------------------------------------------------ exact
class _Plain:
    """The scheme in plain torch, FP64: face by face on the reference's formulas."""

    def __init__(self, m, c, mach, angle, dev):
        t = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device=dev)  # noqa: E731
        self.c, self.dev = c, dev
        X, Y, cells = t(m["x"]), t(m["y"]), t(m["cells"], torch.int64)
        n, nn = cells.shape[0], X.numel()
        tri = cells[:, 3] < 0
        i4 = torch.where(cells < 0, cells[:, :1], cells)
        # edges: corner j to the next corner; a triangle's fourth is left out
        nxt = torch.stack([i4[:, 1], i4[:, 2], torch.where(tri, i4[:, 0], i4[:, 3]), i4[:, 0]], 1)
        own = torch.arange(n, device=dev).repeat_interleave(4).reshape(n, 4)
        use = torch.ones_like(i4, dtype=torch.bool)
        use[:, 3] = ~tri
        key = (torch.minimum(i4, nxt) * nn + torch.maximum(i4, nxt))[use]
        own = own[use]
        uniq, inv = torch.unique(key, return_inverse=True)
        E = uniq.numel()
        c0 = torch.full((E,), n, device=dev).scatter_reduce(0, inv, own, "amin")
        c1 = torch.full((E,), -1, device=dev).scatter_reduce(0, inv, own, "amax")
        # vertex-mean centroids, areas
        nv = torch.where(tri, 3.0, 4.0).double()
        last = torch.where(tri, 0.0, 1.0).double()
        cx = (X[i4[:, :3]].sum(1) + last * X[i4[:, 3]]) / nv
        cy = (Y[i4[:, :3]].sum(1) + last * Y[i4[:, 3]]) / nv

        def area3(p, q, r):
            return 0.5 * (X[p] * (Y[q] - Y[r]) + X[q] * (Y[r] - Y[p]) + X[r] * (Y[p] - Y[q])).abs()

        A = area3(i4[:, 0], i4[:, 1], i4[:, 2]) + last * area3(i4[:, 0], i4[:, 2], i4[:, 3])
        na, nb = uniq // nn, uniq % nn
        ex, ey = 0.5 * (X[na] + X[nb]), 0.5 * (Y[na] + Y[nb])
        dx, dy = X[nb] - X[na], Y[nb] - Y[na]
        L = torch.sqrt(dx * dx + dy * dy)
        nx, ny = -dy / L, dx / L
        sg = torch.where(nx * (ex - cx[c0]) + ny * (ey - cy[c0]) < 0, -1.0, 1.0).double()
        nx, ny = nx * sg, ny * sg
        # boundary edges and their ghosts
        be = t(m["bedges"], torch.int64)
        bk = torch.minimum(be[:, 0], be[:, 1]) * nn + torch.maximum(be[:, 0], be[:, 1])
        bf = torch.searchsorted(uniq, bk)
        B = bf.numel()
        c1 = c1.clone()
        c1[bf] = n + torch.arange(B, device=dev)
        far = torch.tensor([nm == "farfield" for nm in m["names"]], device=dev)[t(m["bpatch"], torch.int64)]
        bt = torch.zeros(E, dtype=torch.int64, device=dev)
        bt[bf] = torch.where(far, 1, 2 if c["wall"] == "slip-wall" else 3)
        o = c0[bf]
        d = torch.sqrt((ex[bf] - cx[o]) ** 2 + (ey[bf] - cy[o]) ** 2)
        cx = torch.cat([cx, ex[bf] + d * nx[bf]])
        cy = torch.cat([cy, ey[bf] + d * ny[bf]])
        self.n, self.B, self.E, self.c0, self.c1, self.bt, self.bf = n, B, E, c0, c1, bt, bf
        self.A, self.L, self.nx, self.ny = A, L, nx, ny
        self.d0 = (ex - cx[c0], ey - cy[c0])
        self.d1 = (ex - cx[c1], ey - cy[c1])
        dij = torch.sqrt((cx[c0] - cx[c1]) ** 2 + (cy[c0] - cy[c1]) ** 2)
        self.geo = torch.sqrt(self.d0[0] ** 2 + self.d0[1] ** 2) / dij
        self.cc = (cx[c1] - cx[c0], cy[c1] - cy[c0])
        t0, t1 = cx[c0] + cx[c1], cy[c0] + cy[c1]
        self.lij = torch.sqrt(t0 * t0 + t1 * t1)
        self.t = (t0 / self.lij, t1 / self.lij)
        self.inner = (bt == 0)
        rho, u, v = _freestream(mach, angle)
        bq = torch.tensor([rho, rho * u, rho * v, 1.0 / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)],
                          dtype=torch.float64, device=dev)
        stop = torch.tensor([1.0, 0.0, 0.0, 1.0 / (GAMMA - 1.0)], dtype=torch.float64, device=dev)
        self.bq = torch.where(far[:, None], bq, stop)  # the ghost state of a wall is not read

    def gather0(self, w):
        """Sum of w (per face) over each cell's faces as its cell 0, and with `minus`, as cell 1."""
        return torch.zeros((self.n + self.B,) + w.shape[1:], dtype=torch.float64, device=self.dev).index_add(0, self.c0, w)

    def pair(self, w0, w1):
        return self.gather0(w0).index_add(0, self.c1, w1)[: self.n]

    @staticmethod
    def pressure(q):
        return (GAMMA - 1.0) * (q[:, 3] - 0.5 / q[:, 0] * (q[:, 1] ** 2 + q[:, 2] ** 2))

    def ghost(self, qL, qb, bt, nx, ny):
        """The far side of each face: mean of both (interior), mirrored, reversed, or characteristic."""
        mean = 0.5 * (qL + qb)
        rV = qL[:, 1] * nx + qL[:, 2] * ny
        slip = torch.stack([qL[:, 0], qL[:, 1] - 2 * rV * nx, qL[:, 2] - 2 * rV * ny, qL[:, 3]], 1)
        wall = torch.stack([qL[:, 0], -qL[:, 1], -qL[:, 2], qL[:, 3]], 1)
        out = torch.where((bt == 0)[:, None], mean, torch.where((bt == 2)[:, None], slip, wall))
        k = (bt == 1).nonzero()[:, 0]
        if k.numel():
            i, b, x, y = qL[k], qb[k], nx[k], ny[k]
            ua, va, pa = b[:, 1] / b[:, 0], b[:, 2] / b[:, 0], self.pressure(b)
            p = self.pressure(i)
            c = torch.sqrt(GAMMA * p / i[:, 0])
            ud, vd = i[:, 1] / i[:, 0], i[:, 2] / i[:, 0]
            rc = i[:, 0] * c
            inl = (i[:, 1] * x + i[:, 2] * y) < 0
            pb = torch.where(inl, 0.5 * (pa + p - rc * (x * (ua - ud) + y * (va - vd))), pa)
            r = torch.where(inl, b[:, 0] + (pb - pa) / (c * c), i[:, 0] + (pb - p) / (c * c))
            u = torch.where(inl, ua - x * (pa - pb) / rc, ud + x * (p - pb) / rc)
            v = torch.where(inl, va - y * (pa - pb) / rc, va + y * (p - pb) / rc)
            sub = torch.stack([r, r * u, r * v, pb / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v)], 1)
            fast = torch.sqrt(i[:, 1] ** 2 + i[:, 2] ** 2) / rc > 1
            sup = torch.where(inl[:, None], b, i)
            out = out.index_copy(0, k, torch.where(fast[:, None], sup, sub))
        return out

    def gradient(self, qf):
        q0, q1 = qf[self.c0], qf[self.c1]
        qR = self.ghost(q0, q1, self.bt, self.nx, self.ny)
        if self.c["gradient"] == "green-gauss":
            g = self.geo[:, None]
            fk = (q0 * (1.0 - g) + qR * g) * self.L[:, None]
            fx, fy = fk * self.nx[:, None], fk * self.ny[:, None]
            return self.pair(fx, -fx) / self.A[:, None], self.pair(fy, -fy) / self.A[:, None]
        dx, dy = self.cc
        one = lambda w: self.pair(w, w)  # noqa: E731
        a00, a01, a11 = one(dx * dx), one(dx * dy), one(dy * dy)
        det = a00 * a11 - a01 * a01
        # cell 1 sees the neighbour at -(dx, dy); both differences change sign, so the products agree
        e0 = q0 - qR
        e1 = torch.where(self.inner[:, None], 0.5 * (q1 - q0), torch.zeros_like(q0))
        sx = self.pair(dx[:, None] * e0, -dx[:, None] * e1)
        sy = self.pair(dy[:, None] * e0, -dy[:, None] * e1)
        return ((a11 / det)[:, None] * sx - (a01 / det)[:, None] * sy,
                (a00 / det)[:, None] * sy - (a01 / det)[:, None] * sx)

    def limit(self, qf, gx, gy):
        n, c0, c1 = self.n, self.c0, self.c1
        use1 = (self.bt < 2)  # a wall's ghost takes the cell's state
        q0, q1 = qf[c0], qf[c1]
        nb = torch.where(use1[:, None], q1, q0)
        hi = lambda red: qf.scatter_reduce(0, c0[:, None].expand(-1, 4), nb, red).scatter_reduce(  # noqa: E731
            0, c1[:, None].expand(-1, 4), q0, red)[:n]
        qmx, qmn = hi("amax"), hi("amin")
        K3 = ((LIM_K * torch.sqrt(self.A)) ** 3)[:, None]

        def side(cell, d, ok):
            i = cell[ok]
            dq = gx[i] * d[0][ok][:, None] + gy[i] * d[1][ok][:, None]
            dmx, dmn, k3 = qmx[i] - qf[i], qmn[i] - qf[i], K3[i]
            D = torch.where(dq > 0, dmx, dmn)
            if self.c["limiter"] == "venkatakrishnan":
                safe = torch.where(dq.abs() > 1e-16, dq, torch.ones_like(dq))
                lim = ((D * D + k3) * safe + 2 * safe * safe * D) / safe / (D * D + 2 * safe * safe + D * safe + k3)
                return i, torch.where(dq.abs() > 1e-16, lim, torch.ones_like(lim))
            s2 = (dmx - dmn) ** 2
            y = s2 / k3 - 1.0
            sig = torch.where(s2 <= k3, torch.ones_like(y),
                              torch.where(s2 <= 2 * k3, 2 * y ** 3 - 3 * y ** 2 + 1, torch.zeros_like(y)))
            safe = torch.where(dq.abs() > 1e-14, dq, torch.ones_like(dq))
            r = torch.where(dq.abs() > 1e-14, D / safe, torch.full_like(D, 2.0))
            lim = torch.where(r >= 2, torch.ones_like(r), -0.25 * r ** 2 + r)
            return i, sig + (1 - sig) * lim

        every = torch.ones_like(self.inner)
        i0, l0 = side(c0, self.d0, every)
        i1, l1 = side(c1, self.d1, self.inner)
        phi = torch.ones((n, 4), dtype=torch.float64, device=self.dev)
        phi = phi.scatter_reduce(0, i0[:, None].expand(-1, 4), l0, "amin")
        return phi.scatter_reduce(0, i1[:, None].expand(-1, 4), l1, "amin")

    def flux(self, qL, qR):
        nx, ny = self.nx, self.ny
        rL, rR = qL[:, 0], qR[:, 0]
        uL, vL, uR, vR = qL[:, 1] / rL, qL[:, 2] / rL, qR[:, 1] / rR, qR[:, 2] / rR
        pL, pR = self.pressure(qL), self.pressure(qR)
        VL, VR = uL * nx + vL * ny, uR * nx + vR * ny
        z = torch.zeros_like(pL)
        f = 0.5 * (VL[:, None] * qL + VR[:, None] * qR
                   + torch.stack([z, pL * nx + pR * nx, pL * ny + pR * ny, VL * pL + VR * pR], 1))
        sL, sR = torch.sqrt(rL), torch.sqrt(rR)
        rho, s = sL * sR, sL + sR
        u, v = (uL * sL + uR * sR) / s, (vL * sL + vR * sR) / s
        h = ((qL[:, 3] + pL) / rL * sL + (qR[:, 3] + pR) / rR * sR) / s
        q2 = u * u + v * v
        c = torch.sqrt((GAMMA - 1.0) * (h - 0.5 * q2))
        V = u * nx + v * ny

        def lam(x):
            a, d = torch.sqrt(x * x + 1e-4), 0.05 * c
            return torch.where(a > d, a, (a * a + d * d) / (2 * d))

        dp, dV, dr = pR - pL, VR - VL, rR - rL
        k1 = lam(V - c) * (dp - rho * c * dV) / (2 * c * c)
        k5 = lam(V + c) * (dp + rho * c * dV) / (2 * c * c)
        k2 = lam(V) * (dr - dp / (c * c))
        k3 = lam(V) * rho
        diss = torch.stack([
            k1 + k2 + k5,
            k1 * (u - c * nx) + k2 * u + k3 * (uR - uL - dV * nx) + k5 * (u + c * nx),
            k1 * (v - c * ny) + k2 * v + k3 * (vR - vL - dV * ny) + k5 * (v + c * ny),
            k1 * (h - c * V) + k2 * q2 * 0.5 + k3 * (u * (uR - uL) + v * (vR - vL) - V * dV) + k5 * (h + c * V)], 1)
        return f - 0.5 * diss

    def laminar(self, qL, qR, gx, gy, mu):
        """Shear and heat terms of the mean state with the face gradient, per face."""
        kh = mu / PR_L
        q = 0.5 * (qL + qR)
        r, u, v, p = q[:, 0], q[:, 1] / q[:, 0], q[:, 2] / q[:, 0], self.pressure(q)

        def parts(g):
            gu, gv = (g[:, 1] - u * g[:, 0]) / r, (g[:, 2] - v * g[:, 0]) / r
            gp = (GAMMA - 1.0) * (g[:, 3] - 0.5 * (g[:, 1] * u + g[:, 2] * v) - 0.5 * r * (u * gu + v * gv))
            return gu, gv, (gp - g[:, 0] * p / r) / r / RGAS

        ux, vx, Tx = parts(gx)
        uy, vy, Ty = parts(gy)
        div = (ux + vy) / 3.0
        xx, yy, xy = 2 * mu * (ux - div), 2 * mu * (vy - div), mu * (uy + vx)
        hx, hy = u * xx + v * xy + kh * Tx, u * xy + v * yy + kh * Ty
        nx, ny = self.nx, self.ny
        return torch.stack([torch.zeros_like(r), nx * xx + ny * xy, nx * xy + ny * yy, nx * hx + ny * hy], 1)

    def residual(self, qk, qm, grads):
        """Flux sums over the area at stage state qk with the gradients and member state of qm."""
        bq = self.bq
        qf = torch.cat([qk, bq])
        if grads is None:
            z = torch.zeros_like(qf)
            gx = gy = z
        else:
            pad = torch.zeros((self.B, 4), dtype=torch.float64, device=self.dev)
            gx, gy = torch.cat([grads[0], pad]), torch.cat([grads[1], pad])
        c0, c1 = self.c0, self.c1
        qL, qR = qf[c0], qf[c1]
        if self.c["second"]:
            phi = torch.cat([self.limit(qf, gx, gy), torch.ones_like(bq)])
            qL = qL + (gx[c0] * self.d0[0][:, None] + gy[c0] * self.d0[1][:, None]) * phi[c0]
            qR = qR + (gx[c1] * self.d1[0][:, None] + gy[c1] * self.d1[1][:, None]) * phi[c1]
        ins = self.inner[:, None]
        f = self.flux(qL, torch.where(ins, qR, self.ghost(qL, qR, self.bt, self.nx, self.ny)))
        if self.c["viscosity"] == "laminar":
            mf = torch.cat([qm, bq])
            gd = (mf[c0] - mf[c1]) / self.lij[:, None]
            bx, by = 0.5 * (gx[c0] + gx[c1]), 0.5 * (gy[c0] + gy[c1])
            t0, t1 = self.t[0][:, None], self.t[1][:, None]
            e = bx * t0 + by * t1 - gd
            lam = self.laminar(qL, qR, bx - e * t0, by - e * t1, self.c["mu"])
            f = f - torch.where(ins, lam, torch.zeros_like(lam))
        fl = f * self.L[:, None]
        return self.pair(-fl, fl) / self.A[:, None]

    def grads(self, q):
        if not self.c["second"] and self.c["viscosity"] == "inviscid":
            return None
        return self.gradient(torch.cat([q, self.bq]))

    def eig_dt(self, q):
        qf = torch.cat([q, self.bq])

        def eig(s):
            V = (s[:, 1] * self.nx + s[:, 2] * self.ny) / s[:, 0]
            return torch.sqrt(GAMMA * self.pressure(s) / s[:, 0]) + V.abs()

        e0 = eig(qf[self.c0])
        e1 = torch.where(self.inner, eig(torch.where(self.inner[:, None], qf[self.c1], qf[self.c0])), e0)
        w = torch.maximum(e0, e1) * self.L
        return (self.c["cfl"] * self.A / self.pair(w, w))[:, None]

    def iterate(self, q):
        dt, g = self.eig_dt(q), self.grads(q)
        qk = q
        for al in (0.25, 0.5, 1.0):
            qk = q + self.residual(qk, q, g) * dt * (al * RELAX)
        return qk


def _wall_forces(P, m, q, mach, angle):
    X = torch.as_tensor(m["x"], dtype=torch.float64, device=P.dev)
    Y = torch.as_tensor(m["y"], dtype=torch.float64, device=P.dev)
    be = torch.as_tensor(m["bedges"], dtype=torch.int64, device=P.dev)
    on = (P.bt[P.bf] >= 2).nonzero()[:, 0]
    e = P.bf[on]
    ex, ey = (0.5 * (Z[be[on, 0]] + Z[be[on, 1]]) for Z in (X, Y))
    cp = 2.0 / (GAMMA * mach * mach) * (P.pressure(q[P.c0[e]]) - 1.0)
    chord = ex.max() - ex.min()
    fx, fy = cp * P.nx[e] * P.L[e] / chord, cp * P.ny[e] * P.L[e] / chord
    xm, ym = ex.min() + 0.25 * chord, ey.mean()
    cm = -((ex - xm) / chord * fy - (ey - ym) / chord * fx).sum()
    sx, sy = fx.sum(), fy.sum()
    ca, sa = math.cos(angle), math.sin(angle)
    return dict(cl=float(-sx * sa + sy * ca), cd=float(sx * ca + sy * sa), cm=float(cm), cp=cp.cpu())


def exact(case, seed):
    """The same in plain torch, 64 bits.  The implicit solver's iterates end at an inexact linear solve: no such value."""
    c = dict(case)
    if c["solver"] == "implicit":
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if c["do"] == "batch":
        out = []
        for k, f in enumerate(_sweep(c["cases"], c["a"], c["b"])):
            cx, cy = meshgen.cell_centroids(f["mesh"])
            P = _Plain(f["mesh"], c, f["mach"], f["aoa_deg"] * DEG, dev)
            q = _flow(torch.from_numpy(cx), torch.from_numpy(cy), f["mach"], f["aoa_deg"] * DEG, seed * 1000 + k)
            q = q.reshape(-1, 4).to(dev)
            for _ in range(c["steps"]):
                q = P.iterate(q)
            out.append(q.reshape(-1).cpu())
        return out
    m = _arrays(c["mesh"], c["a"], c["b"], c["split"], c["fill"])
    cx, cy = meshgen.cell_centroids(m)
    ang = c["aoa"] * DEG
    q = _flow(torch.from_numpy(cx), torch.from_numpy(cy), c["mach"], ang, seed).reshape(-1, 4).to(dev)
    P = _Plain(m, c, c["mach"], ang, dev)
    if c["do"] == "vjp":
        g = torch.Generator().manual_seed(seed)
        v = torch.randn(q.numel(), generator=g, dtype=torch.float64).reshape(-1, 4).to(dev)
        q.requires_grad_(True)
        P.bq = P.bq.clone().requires_grad_(True)
        R = P.residual(q, q, P.grads(q))
        u, b = torch.autograd.grad((R * v).sum(), [q, P.bq])
        return dict(u=u.reshape(-1).cpu(), bq=None)  # (a wall's stored state is not an input of the plain form)
    if c["do"] == "residual":
        return dict(R=P.residual(q, q, P.grads(q)).reshape(-1).cpu())
    for _ in range(c["steps"]):
        q = P.iterate(q)
    out = dict(q=q.reshape(-1).cpu())
    if c["mesh"] != "channel":
        out.update(_wall_forces(P, m, q, c["mach"], ang))
    return out
