"""The work a TILD simulation has this library do, as timed cases over tild.py's entry points.

Every case is a bead-spring system on a grid with its pair styles, driven the way a program drives
it: stepping between log lines, one force evaluation for an outer integrator, an ensemble advanced
as a batch, a serving slot taking its next job, or a log line's observables.  listed() names the
ones that are followed; draw() spreads over the ranges they stand for.  exact() restates the method
in 64-bit torch.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-tild_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tild  # noqa: E402
from tild_systems import ensemble_capacity, ensemble_slot_template  # noqa: E402

PI = math.pi


def _case(name, kind, dim, nx, ny, nz, dx, chains, length, layout, style, order, integrator, steps, **more):
    c = dict(name=name, kind=kind, dim=dim, nx=nx, ny=ny, nz=nz, dx=dx, chains=chains, length=length, layout=layout,
             style=style, order=order, integrator=integrator, steps=steps, solvent=0, fieldphase=False, dt=0.005)
    c.update(more)
    return c


def listed():
    return [
        # a thin film on a small 2D grid, stepped one step per call by a program that looks at the
        # positions after each: launches and latency are all there is
        _case("film_2d_single_steps", "step", 2, 40, 40, 1, 0.5, 200, 10, "diblock", "gaussian", 1, "GJF", 1),
        # the default diblock melt (40,000 beads, 40^3) between two log lines of 100 steps
        _case("diblock_40_log_interval", "step", 3, 40, 40, 40, 0.5, 2000, 20, "diblock", "gaussian", 1, "GJF", 100),
        # the melt of the reference's documentation: 175,000 beads on 45^3, quadratic assignment
        _case("melt_45_order2", "step", 3, 45, 45, 45, 0.5, 7000, 25, "diblock", "gaussian", 2, "GJF", 50),
        # the benchmark's homopolymer blend: 2.6M beads, 128^3, 64-point stencils
        _case("blend_128_order3", "step", 3, 128, 128, 128, 0.5, 130000, 20, "blend", "gaussian_erf", 3, "GJF", 16),
        # polyelectrolyte coacervate: three species and a charge grid, 96^3, Euler-Maruyama
        _case("coacervate_96", "step", 3, 96, 96, 96, 0.5, 8000, 25, "coacervate", "gaussian", 1, "EM", 100,
              solvent=20000, dt=0.002),
        # a lamella guided by a static field in a box that is no cube: odd and unequal edges, erf
        # particles, the highest assignment order
        _case("lamella_odd_order4", "step", 3, 33, 52, 75, 0.4, 2400, 25, "diblock", "erf", 4, "GJF", 32, fieldphase=True),
        # a phase-diagram ensemble of 40 different systems (24^3 to 48^3) advanced together, then read
        _case("ensemble_40", "batch", 3, 24, 48, 0, 0.5, 40, 0, "member", "gaussian", 1, "GJF", 64),
        # a serving slot taking its next job (tables, topology, state), advancing with seven others
        _case("serve_next_job", "serve", 3, 24, 45, 0, 0.5, 8, 0, "member", "gaussian", 1, "GJF", 32),
        # one force evaluation for an outer integrator that hands over its positions: homopolymer in
        # solvent is not a pair of species but three, cubic assignment, odd edges
        _case("forces_63_outer_loop", "forces", 3, 63, 63, 63, 0.5, 12000, 20, "ternary", "gaussian_erf", 3, "GJF", 1,
              solvent=8000),
        # the log line of the charged system: energies, virials, bonds
        _case("log_line_96", "observables", 3, 96, 96, 96, 0.5, 8000, 25, "coacervate", "gaussian", 1, "EM", 1,
              solvent=20000, dt=0.002),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["forces", "observables", "batch", "serve"])
    if kind in ("batch", "serve"):
        lo = rng.randint(24, 40)
        n = rng.randint(4, 40) if kind == "batch" else rng.randint(2, 8)
        return _draw_done(dict(kind=kind, nx=lo, ny=rng.randint(lo, 48), chains=n, layout="member",
                               steps=rng.choice([8, 24, 32, 64])))
    dim = 2 if rng.random() < 0.2 else 3
    base = math.exp(rng.uniform(math.log(16), math.log(104 if dim == 3 else 200)))
    edge = [max(12, min(128 if dim == 3 else 200, int(base * rng.uniform(0.8, 1.25)))) for _ in range(3)]
    if rng.random() < 0.4:
        edge = [edge[0]] * 3  # cubes are common
    if dim == 2:
        edge[2] = 1
    order = rng.choice([1, 1, 2, 3, 4])
    layout = rng.choice(["diblock", "diblock", "blend", "coacervate", "ternary", "homopolymer"])
    points = edge[0] * edge[1] * edge[2]
    length = rng.randint(5, 40)
    beads = min(points * math.exp(rng.uniform(math.log(0.25), math.log(1.9))), 1.2e6)
    chains = max(2, int(beads / length)) // 2 * 2
    solvent = int(0.1 * beads) if layout in ("coacervate", "ternary") else 0
    steps = rng.choice([1, 20, 32, 50, 100]) if points < 200000 else rng.choice([16, 20, 32])
    return _draw_done(dict(kind=kind, dim=dim, nx=edge[0], ny=edge[1], nz=edge[2], dx=rng.choice([0.5, 0.5, 0.4, 0.6]),
                           chains=chains, length=length, layout=layout, solvent=solvent, order=order,
                           style=rng.choice(["gaussian", "gaussian", "gaussian_erf", "erf"]),
                           integrator=rng.choice(["GJF", "GJF", "EM"]), steps=steps if kind == "step" else 1,
                           fieldphase=layout == "diblock" and dim == 3 and rng.random() < 0.25,
                           dt=rng.choice([0.002, 0.005])))


def _draw_done(got):
    c = _case("", "step", 3, 0, 0, 0, 0.5, 0, 0, "", "gaussian", 1, "GJF", 1)
    del c["name"]
    c.update(got)
    return c


# ---- systems ----------------------------------------------------------------------------------
def _system(case, seed):
    rng = np.random.default_rng([seed, 11])
    dim = case["dim"]
    nx = [case["nx"], case["ny"], case["nz"]]
    box = [float(np.float32(n * case["dx"])) for n in nx[:dim]]
    L = np.asarray(box, np.float32)
    N, n_chains, ns_chain = case["length"], case["chains"], case["chains"] * case["length"]
    # chains: Gaussian random walks from uniform starts, wrapped into [0, L)
    x = rng.standard_normal((n_chains, N, dim), dtype=np.float32) * np.float32(1.0 / math.sqrt(dim))
    x[:, 0] = rng.random((n_chains, dim), dtype=np.float32) * L
    x = np.cumsum(x, axis=1, dtype=np.float32).reshape(-1, dim)
    x = np.concatenate([x, rng.random((case["solvent"], dim), dtype=np.float32) * L])
    x -= np.floor(x / L) * L
    x = np.where((x >= L) | (x < 0), np.float32(0), x)
    ns = x.shape[0]
    layout = case["layout"]
    chain = np.arange(ns_chain) // N
    if layout == "homopolymer":
        types, ntypes = np.zeros(ns, np.int32), 1
    elif layout == "diblock":
        types, ntypes = (np.arange(ns_chain) % N >= N // 2).astype(np.int32), 2
    else:  # chains of two species; coacervates and ternary blends have a solvent too
        types, ntypes = (chain % 2).astype(np.int32), 2
        if layout in ("coacervate", "ternary"):
            types, ntypes = np.concatenate([types, np.full(case["solvent"], 2, np.int32)]), 3
    charges = None
    if layout == "coacervate":
        charges = np.where(types == 2, 0.0, np.where(types == 0, 1.0, -1.0)).astype(np.float32)
    # linear bonds, stored from both ends
    i = np.arange(ns)
    at, inside = i % N, i < ns_chain
    prev, nxt = inside & (at > 0), inside & (at < N - 1)
    n_bonds = prev.astype(np.int32) + nxt
    bonded = np.zeros((ns, 3), np.int32)
    bonded[:, 0] = np.where(prev, i - 1, np.where(nxt, i + 1, 0))
    bonded[:, 1] = np.where(prev & nxt, i + 1, 0)
    rho0 = ns / float(np.prod([float(v) for v in box]))
    kind = {"gaussian": tild.STYLE_GAUSSIAN, "erf": tild.STYLE_ERF, "gaussian_erf": tild.STYLE_GAUSSIAN_ERF}[case["style"]]
    sigma, rp = (math.sqrt(0.5), 0.0) if case["style"] == "gaussian" else (0.5, 0.5)
    styles = [tild.Style(kind, a, b, (25.0 if a == b else 51.0) / rho0, sigma, rp)
              for a in range(ntypes) for b in range(a, ntypes)]
    if case["fieldphase"]:
        styles.append(tild.Style(tild.STYLE_FIELDPHASE, 0, 1, 0.5 / rho0, phase=0, dir=2, n_periods=2))
    integ = tild.INTEGRATOR_GJF if case["integrator"] == "GJF" else tild.INTEGRATOR_EM
    return tild.System(dim=dim, nx=nx, box=box + [1.0] * (3 - dim), types=types, x=x, n_bonds=n_bonds, bonded_to=bonded,
                       bond_type=np.zeros((ns, 3), np.int32), ntypes=ntypes, styles=styles, bond_k=(1.5,),
                       bond_req=(0.0,), integrators=[(integ, -1)], pmeorder=case["order"], delt=case["dt"],
                       seed=12345 + seed % 100000, charges=charges, bjerrum=1.0, smearing=0.5)


def _edge(case, k):
    """Grid edge of the k-th ensemble member: the range is covered evenly."""
    return case["nx"] + k * (case["ny"] - case["nx"]) // max(1, case["chains"] - 1)


def _member(case, seed, k):
    """The k-th member: density 5, chain lengths 10 to 40 across the ensemble."""
    g, N = _edge(case, k), 10 + 7 * k % 31
    chains = max(1, round(5.0 * (0.5 * g) ** 3 / N))
    return _system(dict(case, dim=3, nx=g, ny=g, nz=g, chains=chains, length=N, layout="diblock"), 64 * seed + k)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.turn = case, 0
    if case["kind"] == "batch":
        s.batch = tild.Batch([_member(case, seed, k) for k in range(case["chains"])])
    elif case["kind"] == "serve":
        edges = [_edge(case, k) for k in range(case["chains"])]
        s.batch = tild.Batch([ensemble_slot_template(g) for g in edges], capacity=[ensemble_capacity(g) for g in edges])
        s.jobs = [_member(case, seed, k) for k in range(case["chains"])]
    else:
        s.system = _system(case, seed)
        s.ctx = tild.Context(s.system)
        if case["kind"] == "step":
            s.frame = torch.empty((s.system.ns, s.system.dim), pin_memory=True).numpy()
        elif case["kind"] == "observables":
            s.ctx.forces()
    return s


def run(s):
    kind, steps = s.case["kind"], s.case["steps"]
    if kind == "step":  # steps up to the next frame, and the frame's positions
        s.ctx.step(steps)
        s.ctx.snapshot_wait(s.ctx.snapshot_async(s.frame, None))
        return s.frame
    if kind == "batch":  # the morphologies: every member's densities
        s.batch.step(steps)
        return [s.batch.density(k) for k in range(len(s.batch.systems))]
    if kind == "serve":  # the next job takes its slot; its positions are read when it is due
        k = s.turn % len(s.jobs)
        s.turn += 1
        s.batch.load(k, s.jobs[k])
        s.batch.step(steps)
        return s.batch.get_state(k)[0]
    if kind == "forces":
        s.ctx.set_state(s.system.x)
        return s.ctx.forces()
    o = s.ctx.observables()
    del o["step"]
    return o


def work(case):
    """Each array once per step: beads 104 B with GJF and 64 B with EM in 3D, and per node and channel
    a density written, its spectrum both ways, the D fields both ways and their gather (48 B in 3D);
    2.5 M log2(M) operations for each of the 1 + D real transforms of a channel, and 2 + 2 D per
    stencil point of a bead.  Positions or forces that are read back are counted once."""
    if case["kind"] in ("batch", "serve"):
        n = case["chains"]
        edges = [_edge(case, k) for k in range(n)]
        beads, points, ch, dim, order = sum(5.0 * (0.5 * g) ** 3 for g in edges), sum(float(g) ** 3 for g in edges), 2, 3, 1
        out = 8.0 * points if case["kind"] == "batch" else 12.0 * beads / n
    else:
        dim, order = case["dim"], case["order"]
        beads = float(case["chains"] * case["length"] + case["solvent"])
        points = float(case["nx"] * case["ny"] * (case["nz"] if dim == 3 else 1))
        ch = {"homopolymer": 1, "diblock": 2, "blend": 2, "ternary": 3, "coacervate": 4}[case["layout"]]
        out = 4.0 * dim * beads
    if case["kind"] == "observables":
        types = 3 if ch == 4 else ch
        pairs = types * (types + 1) // 2
        return {"bytes": 32.0 * beads + points * (4.0 * ch + pairs * (2.0 + 4.0 * (6 if dim == 3 else 3))),
                "flops": points * pairs * 20.0 + 30.0 * beads}
    per_bead = (104.0 if case["integrator"] == "GJF" else 64.0) * dim / 3
    step_bytes = beads * per_bead + points * ch * (12.0 + 12.0 * dim)
    step_flops = points * ch * (1 + dim) * 2.5 * math.log2(points) + beads * (order + 1) ** dim * (2 + 2 * dim)
    return {"bytes": case["steps"] * step_bytes + out, "flops": case["steps"] * step_flops}


# ---- the same in 64 bits ----------------------------------------------------------------------
_MASK = 0xFFFFFFFF


def _mulhilo(a, b):
    """High and low 32 bits of the product of a constant and a tensor of 32-bit values (int64)."""
    lo_part, hi_part = (b & 0xFFFF) * a, (b >> 16) * a
    mid = hi_part + (lo_part >> 16)
    return (mid >> 16) & _MASK, ((mid << 16) | (lo_part & 0xFFFF)) & _MASK


def _normals(seed, beads, step, dev):
    """The three normals of each bead at a step: Philox4x32-10 keyed by bead and seed, Box-Muller."""
    c = [torch.full_like(beads, step & _MASK), torch.full_like(beads, step >> 32), torch.zeros_like(beads),
         torch.full_like(beads, (seed >> 32) & _MASK)]
    k0, k1 = beads.clone(), seed & _MASK
    for _ in range(10):
        h0, l0 = _mulhilo(0xD2511F53, c[0])
        h1, l1 = _mulhilo(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & _MASK, (k1 + 0xBB67AE85) & _MASK
    u = [((v >> 8) | (1 if j % 2 == 0 else 0)).double() * 2.0 ** -24 for j, v in enumerate(c)]
    r0, r1 = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
    return torch.stack([r0 * torch.cos(2 * PI * u[1]), r0 * torch.sin(2 * PI * u[1]), r1 * torch.cos(2 * PI * u[3])], 1)


class _Exact:
    """One system in 64 bits: the same constants (grid spacing, time step and so on are the 32-bit
    numbers that the library is given), every sum and function in double."""

    def __init__(self, s):
        self.s = s
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.D, self.n = s.dim, [int(v) for v in s.nx[:s.dim]]
        L32 = [np.float32(v) for v in s.box[:s.dim]]
        self.L = [float(v) for v in L32]
        self.Lh = [float(np.float32(0.5) * v) for v in L32]
        self.dx = [float(v / np.float32(m)) for v, m in zip(L32, self.n)]
        gv = np.float32(1)
        for v, m in zip(L32, self.n):
            gv = gv * (v / np.float32(m))
        self.gvol, self.M, self.dV, self.V = float(gv), math.prod(self.n), math.prod(self.dx), math.prod(self.L)
        self.P = s.pmeorder
        self.types = torch.as_tensor(s.types, dtype=torch.int64, device=self.dev)
        self.q = None if s.charges is None else torch.as_tensor(s.charges, dtype=torch.float64, device=self.dev)
        self.x = torch.as_tensor(s.x, dtype=torch.float64, device=self.dev)
        self.xo, self.noise, self.step_count = self.x.clone(), torch.zeros_like(self.x), 0
        self.nch = s.ntypes + (0 if self.q is None else 1)
        # wave vectors, axis order (z, y, x) as the grids are stored; the Nyquist derivative is 0
        self.k, self.kd = [], []
        for d in range(self.D):
            m = torch.arange(self.n[d], dtype=torch.float64, device=self.dev)
            m = torch.where(m < self.n[d] / 2, m, m - self.n[d])
            kv = 2 * PI * m / self.L[d]
            kd = kv.clone()
            if self.n[d] % 2 == 0:
                kd[self.n[d] // 2] = 0
            shape = [1] * self.D
            shape[self.D - 1 - d] = self.n[d]
            self.k.append(kv.reshape(shape))
            self.kd.append(kd.reshape(shape))
        self.k2 = sum(v * v for v in self.k)
        self.u = [self._u(st) for st in s.styles]
        b = torch.as_tensor(s.bonded_to, dtype=torch.int64, device=self.dev)
        nb = torch.as_tensor(s.n_bonds, dtype=torch.int64, device=self.dev)
        bt = torch.as_tensor(s.bond_type, dtype=torch.int64, device=self.dev)
        self.ends = []
        for j in range(3):
            i = torch.nonzero(nb > j).reshape(-1)
            if len(i):
                kk = torch.as_tensor([float(np.float32(v)) for v in s.bond_k], dtype=torch.float64, device=self.dev)
                rr = torch.as_tensor([float(np.float32(v)) for v in s.bond_req], dtype=torch.float64, device=self.dev)
                self.ends.append((i, b[i, j], kk[bt[i, j]], rr[bt[i, j]]))

    def _u(self, st):
        if st.kind == tild.STYLE_FIELDPHASE:
            return None
        A, s2, R = float(np.float32(st.prefactor)), float(np.float32(st.sigma)) ** 2, float(np.float32(st.rp))
        k2 = self.k2
        g = A * torch.exp(-0.5 * k2 * s2)
        if st.kind == tild.STYLE_GAUSSIAN:
            return g
        k = torch.sqrt(k2)
        t = 4 * PI * (torch.sin(R * k) - R * k * torch.cos(R * k)) / torch.where(k2 == 0, 1.0, k2 * k)
        t = torch.where(k2 == 0, 4 * PI * R ** 3 / 3, t)
        return g * t * t if st.kind == tild.STYLE_ERF else g * t

    def _stencil(self):
        """Node indices and weights per axis: nearest node for even orders, containing cell for odd."""
        idx, W = [], []
        for d in range(self.D):
            xd, h = self.x[:, d], self.dx[d]
            gi = torch.floor((xd + 0.5 * h) / h) if self.P % 2 == 0 else torch.floor(xd / h)
            sx = (xd - gi * h if self.P % 2 == 0 else xd - (gi + 0.5) * h) / h
            s2 = sx * sx
            if self.P == 1:
                w = [0.5 - sx, 0.5 + sx]
            elif self.P == 2:
                w = [0.125 - 0.5 * sx + 0.5 * s2, 0.75 - s2, 0.125 + 0.5 * sx + 0.5 * s2]
            elif self.P == 3:
                s3 = s2 * sx
                w = [(1 - 6 * sx + 12 * s2 - 8 * s3) / 48, (23 - 30 * sx - 12 * s2 + 24 * s3) / 48,
                     (23 + 30 * sx - 12 * s2 - 24 * s3) / 48, (1 + 6 * sx + 12 * s2 + 8 * s3) / 48]
            else:  # the method's order 4 takes the fourth power in the cubic terms
                s4 = s2 * s2
                w = [(1 - 8 * sx + 24 * s2 - 32 * s4 + 16 * s4) / 384, (19 - 44 * sx + 24 * s2 + 16 * s4 - 16 * s4) / 96,
                     (115 - 120 * s2 + 48 * s4) / 192, (19 + 44 * sx + 24 * s2 - 16 * s4 - 16 * s4) / 96,
                     (1 + 8 * sx + 24 * s2 + 32 * s4 + 16 * s4) / 384]
            base = gi.long() - self.P // 2
            idx.append([(base + a) % self.n[d] for a in range(self.P + 1)])
            W.append(w)
        for a in np.ndindex(*([self.P + 1] * self.D)):
            m, w = 0, 1.0
            for d in reversed(range(self.D)):
                m = m * self.n[d] + idx[d][a[d]]
                w = w * W[d][a[d]]
            yield m, w

    def density(self):
        rho = torch.zeros(self.nch * self.M, dtype=torch.float64, device=self.dev)
        for m, w in self._stencil():
            rho.index_add_(0, self.types * self.M + m, w / self.gvol)
            if self.q is not None:
                rho.index_add_(0, self.s.ntypes * self.M + m, w * self.q / self.gvol)
        return rho.reshape([self.nch] + self.n[::-1])

    def forces(self):
        s, ax = self.s, tuple(range(1, self.D + 1))
        rho = self.density()
        rk = torch.fft.fftn(rho, dim=ax)
        phi = torch.zeros_like(rk)
        for st, u in zip(s.styles, self.u):
            if u is not None:
                phi[st.type1] += u * rk[st.type2]
                phi[st.type2] += u * rk[st.type1]
        if self.q is not None:
            a2 = float(np.float32(s.smearing)) ** 2
            k2 = torch.where(self.k2 == 0, 1.0, self.k2)
            e = 4 * PI * float(np.float32(s.bjerrum)) / k2 * torch.exp(-k2 / a2)
            phi[s.ntypes] = torch.where(self.k2 == 0, 0.0, e) * rk[s.ntypes]
        field = [torch.fft.ifftn(-1j * self.kd[d] * phi, dim=ax).real for d in range(self.D)]
        for st in s.styles:
            if st.kind == tild.STYLE_FIELDPHASE:  # lamellae along one axis
                d = st.dir
                r = torch.arange(self.n[d], dtype=torch.float64, device=self.dev) * self.dx[d]
                a = 2 * PI * st.n_periods / self.L[d]
                shape = [1] * self.D
                shape[self.D - 1 - d] = self.n[d]
                f = (float(np.float32(st.prefactor)) * a * torch.cos(a * r)).reshape(shape)
                field[d][st.type1] += rho[st.type1] * f
                field[d][st.type2] -= rho[st.type2] * f
        flat = [f.reshape(-1) for f in field]
        f = torch.zeros_like(self.x)
        for m, w in self._stencil():
            for d in range(self.D):
                f[:, d] += w * flat[d][self.types * self.M + m]
                if self.q is not None:
                    f[:, d] += w * self.q * flat[d][s.ntypes * self.M + m]
        for i, j, k, r0 in self.ends:
            dr = self._image(self.x[i] - self.x[j])
            r2 = (dr * dr).sum(1)
            r = torch.sqrt(torch.where(r2 > 1e-4, r2, 1.0))
            mf = torch.where(r2 > 1e-4, 2 * k * (r - r0) / r, 0.0)
            f.index_add_(0, i, -mf[:, None] * dr)
        return f

    def _image(self, dr):
        L, Lh = (torch.tensor(v, dtype=torch.float64, device=self.dev) for v in (self.L, self.Lh))
        return torch.where(dr > Lh, dr - L, torch.where(dr < -Lh, dr + L, dr))

    def step(self):
        s = self.s
        f = self.forces()
        dt = float(np.float32(s.delt))
        amp = float(np.sqrt(np.float32(2.0) * np.float32(s.delt), dtype=np.float32))
        ids = torch.arange(s.ns, dtype=torch.int64, device=self.dev)
        z = amp * _normals(s.seed, ids, self.step_count + 1, self.dev)[:, :self.D]
        L = torch.tensor(self.L, dtype=torch.float64, device=self.dev)
        if s.integrators[0][0] == tild.INTEGRATOR_GJF:  # unit masses and diffusivities
            b = 1 / (1 + dt / 2)
            a = (1 - dt / 2) / (1 + dt / 2)
            gap = self.xo - self.x
            xo = self.xo - torch.where(gap > L / 2, L, 0.0) + torch.where(gap < -L / 2, L, 0.0)
            xn = 2 * b * self.x - a * xo + b * dt * dt * f + b * dt / 2 * (z + self.noise)
            self.xo, self.noise = self.x, z
        else:
            xn = self.x + dt * f + z
        self.x = torch.where(xn > L, xn - L, torch.where(xn < 0, xn + L, xn))
        self.step_count += 1

    def observables(self):
        s, D = self.s, self.D
        rk = torch.fft.fftn(self.density(), dim=tuple(range(1, D + 1)))
        pairs = [(0, 0), (1, 1), (2, 2), (1, 0), (2, 0), (2, 1)] if D == 3 else [(0, 0), (1, 1), (1, 0)]
        energy, virial = [], []
        for st, u in zip(s.styles, self.u):
            if u is None:
                energy.append(0.0)
                virial.append([0.0] * len(pairs))
                continue
            c = rk[st.type2] * rk[st.type1].conj()
            energy.append(float((u * c).sum().real) * self.dV / self.M)
            fr = [torch.fft.ifftn(-1j * self.kd[d] * u).real * self.M for d in range(D)]
            row = []
            for al, be in pairs:
                h32, L32 = np.float32(self.dx[al]), np.float32(self.L[al])
                r = np.arange(self.n[al], dtype=np.float32) * h32
                r = np.where(r > np.float32(self.Lh[al]), r - L32, r).astype(np.float64)
                shape = [1] * D
                shape[D - 1 - al] = self.n[al]
                vk = torch.fft.fftn(torch.as_tensor(r, device=self.dev).reshape(shape) * fr[be]) / self.M ** 2
                row.append(float((vk * c).sum().real) * self.dV / self.V / D)
            virial.append(row)
        uelec = 0.0
        if self.q is not None:
            a2 = float(np.float32(s.smearing)) ** 2
            k2 = torch.where(self.k2 == 0, 1.0, self.k2)
            e = torch.where(self.k2 == 0, 0.0, 4 * PI * float(np.float32(s.bjerrum)) / k2 * torch.exp(-k2 / (2 * a2)))
            uelec = float((e * rk[s.ntypes].abs() ** 2).sum()) / self.M
        ub, bv = 0.0, [0.0] * len(pairs)
        for i, j, k, r0 in self.ends:
            once = j > i
            dr = self._image(self.x[i] - self.x[j])[once]
            r = torch.sqrt((dr * dr).sum(1))
            ub += float((k[once] * (r - r0[once]) ** 2).sum())
            mf = 2 * k[once] * (r - r0[once]) / r
            for c, (al, be) in enumerate(pairs):
                bv[c] += float((-mf * dr[:, al] * dr[:, be]).sum()) / self.V / D
        energy, virial, bv = np.array(energy), np.array(virial).reshape(len(energy), len(pairs)), np.array(bv)
        return {"upe": float(energy.sum()) + uelec + ub, "ubond": ub, "uelec": uelec, "ptens": virial.sum(0) + bv,
                "bond_vir": bv, "style_energy": energy, "style_virial": virial}


def _advanced(system, steps, density=False):
    e = _Exact(system)
    for _ in range(steps):
        e.step()
    return e.density().reshape(e.nch, e.M) if density else e.x


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "batch":  # densities belong to the last force evaluation, before the last update
        return [_advanced(_member(case, seed, k), steps - 1, True) for k in range(case["chains"])]
    if kind == "serve":
        return _advanced(_member(case, seed, 0), steps)
    s = _system(case, seed)
    if kind == "step":
        return _advanced(s, steps)
    return _Exact(s).forces() if kind == "forces" else _Exact(s).observables()
