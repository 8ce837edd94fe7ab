"""The work a user of this framework has it do, as cases that can be timed.

Five kinds of pass, each through the public handle (`parm_gb300.System`) and, for whole Atom records, the C ABI's
parm_set_atoms / parm_get_atoms on page-locked host memory:

* verlet   -- NVE Lennard-Jones: some CollectionVerlet steps of a running simulation, then the records come back;
* langevin -- a batch of WCA replicas under CollectionSol, the same way;
* damped   -- a soft-sphere configuration from the host relaxed by CollectionDamped (new positions every pass);
* cg       -- a batch of soft-sphere configurations from the host, some CollectionNLCGV minimiser steps each;
* analyse  -- frames of a stored trajectory: list, forces, energy, virial, stress and contacts of host positions.

A pass returns the whole state in the caller's atom order.  FP64 handles return it in float64.  Mixed-precision handles
hold pair forces in FP32, so their forces, velocities and displacements since the start come back as float32 (formed on
the GPU by torch from the records read back, as an analysis in torch does).
"""
import itertools
import math

import numpy as np
import torch

from parm_gb300 import System, capi

SIGP = 2.0 ** (-1.0 / 6.0)          # the conventional LJ length in units of the minimum's position
CUT = 2.5 * SIGP
CG = [0.1, 0.0, 1.0, 1000.0, 10.0, 1e-4, 0.0, 0.0, 0.0, 0.0, 0.0]   # CollectionNLCGV's defaults with dt = 0.1
DAMPING = 1.0


def listed():
    return [
        # the reference's own LJ program size, bit-exact path: every launch is latency
        dict(name="lj1000_fp64", kind="verlet", prec="fp64", nx=10, ny=10, nz=10, steps=64, dt=0.001, skin=0.4),
        # an ordinary FP64 simulation, ragged box
        dict(name="lj30k_fp64", kind="verlet", prec="fp64", nx=31, ny=33, nz=29, steps=16, dt=0.002, skin=0.3),
        # the benchmark's box on the FP64 path, the largest FP64 run
        dict(name="lj1m_fp64", kind="verlet", prec="fp64", nx=128, ny=128, nz=64, steps=4, dt=0.002, skin=0.3),
        # a small and an ordinary mixed-precision simulation
        dict(name="lj4k_mixed", kind="verlet", prec="mixed", nx=16, ny=17, nz=15, steps=64, dt=0.002, skin=0.3),
        dict(name="lj30k_mixed", kind="verlet", prec="mixed", nx=31, ny=33, nz=29, steps=64, dt=0.002, skin=0.3),
        # the headline benchmark: 1,048,576 LJ atoms
        dict(name="lj1m_mixed", kind="verlet", prec="mixed", nx=128, ny=128, nz=64, steps=32, dt=0.002, skin=0.3),
        # batched WCA Langevin replicas of 256 to 32768 atoms
        dict(name="replicas_mixed", kind="langevin", prec="mixed", nsys=48, nmin=256, nmax=32768, steps=16, dt=0.001,
             skin=0.3),
        # one bidisperse 3D packing of Hertzian-like spheres (exponent 2.5), damped relaxation on the FP64 path
        dict(name="spheres5k_fp64", kind="damped", prec="fp64", nd=3, nsys=1, nmin=5003, nmax=5003, phi=0.64,
             expo=2.5, steps=32, dt=0.05, skin=0.1),
        # 2D harmonic disks, damped relaxation, mixed
        dict(name="disks20k_mixed", kind="damped", prec="mixed", nd=2, nsys=1, nmin=20011, nmax=20011, phi=0.84,
             expo=2.0, steps=64, dt=0.05, skin=0.1),
        # 65,536 harmonic disks at phi = 0.84 under the conjugate-gradient minimiser, FP64 phase
        dict(name="disks65k_cg_fp64", kind="cg", prec="fp64", nd=2, nsys=1, nmin=65536, nmax=65536, phi=0.84,
             expo=2.0, steps=4, skin=0.3),
        # a batch of 3D packings of 64 to 4096 spheres under the minimiser, mixed phase
        dict(name="packings_cg_mixed", kind="cg", prec="mixed", nd=3, nsys=48, nmin=64, nmax=4096, phi=0.64,
             expo=2.5, steps=4, skin=0.3),
        # frames of a stored LJ trajectory
        dict(name="analyse131k_mixed", kind="analyse", prec="mixed", nx=64, ny=64, nz=32, skin=0.3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice(rng, lo, hi):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nx = max(9, int(n ** (1.0 / 3.0) * rng.uniform(0.85, 1.3)))
    ny = max(9, int(n ** (1.0 / 3.0) * rng.uniform(0.85, 1.15)))
    return nx, ny, max(9, int(n / (nx * ny)))


def draw(rng):
    kind = rng.choice(["verlet", "verlet", "langevin", "damped", "cg", "analyse"])
    prec = rng.choice(["fp64", "mixed"])
    if kind in ("verlet", "analyse"):
        nx, ny, nz = _lattice(rng, 900, 900_000 if kind == "verlet" else 400_000)
        c = dict(kind=kind, prec=prec, nx=nx, ny=ny, nz=nz, skin=round(rng.uniform(0.2, 0.45), 3))
        if kind == "verlet":
            most = (4e6 if prec == "fp64" else 3e7) / (nx * ny * nz)
            c.update(steps=max(2, min(64, int(most * rng.uniform(0.4, 1.0)))), dt=rng.choice([0.001, 0.002]))
        return c
    if kind == "langevin":
        nmax = _log_int(rng, 1000, 32768)
        nsys = max(1, min(64, int(300_000 / nmax * rng.uniform(0.2, 1.5))))
        return dict(kind=kind, prec=prec, nsys=nsys, nmin=256, nmax=nmax, steps=rng.randint(4, 16), dt=0.001,
                    skin=round(rng.uniform(0.2, 0.45), 3))
    nd = rng.choice([2, 3])
    nmax = _log_int(rng, 700, 60_000 if nd == 2 else 20_000)
    nsys = 1 if rng.random() < 0.5 else max(1, min(64, int(60_000 / nmax)))
    c = dict(kind=kind, prec=prec, nd=nd, nsys=nsys, nmin=nmax if nsys == 1 else 64, nmax=nmax,
             phi=0.84 if nd == 2 else 0.64, expo=rng.choice([2.0, 2.5]), steps=rng.randint(2, 4))
    if kind == "damped":
        c.update(steps=rng.randint(16, 64), dt=0.05, skin=0.1)
    else:
        c.update(skin=0.3)
    return c


# ---------------------------------------------------------------------------
# inputs (NumPy, from the seed alone)
# ---------------------------------------------------------------------------
def _inputs(c, seed):
    """sizes, nd, box sides (nsys, nd), positions, velocities, pair kind, parameters (n, 3), list skin."""
    rng = np.random.default_rng([seed, 77])
    if c["kind"] in ("verlet", "analyse"):
        # simple-cubic lattice at density 0.8 in LJ units, jittered, Maxwell velocities at T = 1
        a = (SIGP ** 3 / 0.8) ** (1.0 / 3.0)
        shape = (c["nx"], c["ny"], c["nz"])
        g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3)
        amp = 0.05 if c["kind"] == "verlet" else 0.12   # a frame of a running simulation is a liquid
        x = (g + 0.5) * a + rng.uniform(-amp * SIGP, amp * SIGP, size=g.shape)
        v = rng.normal(size=g.shape)
        v -= v.mean(axis=0)
        prm = np.tile([1.0, 1.0, CUT], (len(x), 1))
        return [len(x)], 3, np.array([[k * a for k in shape]]), x, v, capi.LJCUT, prm, c["skin"] * SIGP
    # the sizes of a batch belong to the case; the configurations to the seed
    srng = np.random.default_rng([c["nsys"], c["nmin"], c["nmax"]])
    sizes = np.exp(srng.uniform(np.log(c["nmin"]), np.log(c["nmax"] + 0.5), size=c["nsys"])).astype(int)
    xs, ps, Ls = [], [], []
    if c["kind"] == "langevin":
        for N in sizes:
            side = (N / (srng.uniform(0.5, 0.9) / SIGP ** 3)) ** (1.0 / 3.0)
            k = int(np.ceil(N ** (1.0 / 3.0)))
            g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:N]
            xs.append((g + 0.5 + rng.uniform(-0.05, 0.05, size=(N, 3))) * (side / k))
            ps.append(np.tile([1.0, 1.0, 0.0], (N, 1)))
            Ls.append([side] * 3)
        x = np.concatenate(xs)
        return sizes.tolist(), 3, np.array(Ls), x, rng.normal(size=x.shape), capi.LJREPULSE, np.concatenate(ps), \
            c["skin"] * SIGP
    nd = c["nd"]
    for N in sizes:   # bidisperse 1 : 1.4 spheres (disks), random
        sig = np.where(np.arange(N) < N // 2, 1.0, 1.4)
        vol = np.sum(np.pi * sig ** 3 / 6) if nd == 3 else np.sum(np.pi * sig ** 2 / 4)
        side = (vol / c["phi"]) ** (1.0 / nd)
        xs.append(rng.uniform(0, side, size=(N, nd)))
        ps.append(np.stack([np.ones(N), sig, np.full(N, c["expo"])], 1))
        Ls.append([side] * nd)
    x = np.concatenate(xs)
    return sizes.tolist(), nd, np.array(Ls), x, np.zeros_like(x), capi.REPULSION, np.concatenate(ps), c["skin"]


# ---------------------------------------------------------------------------
# the framework
# ---------------------------------------------------------------------------
class _State:
    """A handle with its simulation set up, and page-locked records {x, v, a, f, m} for its atoms."""

    def __init__(self, c, seed):
        self.c, self.seed = c, seed
        sizes, nd, L, x, v, kind, prm, skin = _inputs(c, seed)
        n = len(x)
        self.nd, self.mixed = nd, c["prec"] == "mixed"
        g = self.g = System(sizes, ndim=nd, precision=c["prec"])
        g.set_boxes(L)
        g.set_atoms(x=x, v=v, a=np.zeros_like(x), f=np.zeros_like(x), m=np.ones(n))
        g.set_interaction(kind, prm, skin)
        g.nlist_update(False)
        g.set_forces(True)
        g.nlist_update(False)
        self.out = torch.zeros((n, g.stride), dtype=torch.float64, pin_memory=torch.cuda.is_available())
        self.frames, self.turn = [], 0
        if c["kind"] in ("damped", "cg", "analyse"):
            # host configurations a pass starts from (analyse: two frames further apart than the list's skin)
            far = np.zeros_like(x)
            if c["kind"] == "analyse":
                far = np.random.default_rng([seed, 78]).normal(scale=0.05, size=x.shape) + 0.6 * skin
            for k in range(2 if c["kind"] == "analyse" else 1):
                rec = torch.zeros((n, g.stride), dtype=torch.float64, pin_memory=torch.cuda.is_available())
                rec[:, :nd] = torch.from_numpy(x + k * far)
                rec[:, 4 * nd] = 1.0
                self.frames.append(rec)
        self.x0 = torch.from_numpy(x)
        if self.mixed and torch.cuda.is_available():
            self.x0 = self.x0.cuda()
        if c["kind"] == "cg":
            g.nlcg_init(np.array(CG), boxed=False)
            g.nlcg_reset()

    def upload(self, rec):
        capi.check(self.g.lib.parm_set_atoms(self.g.h, capi.dptr(rec.numpy()), self.g.stride, 31))

    def records(self):
        """The handle's records as (displacement or position, velocity, acceleration, force)."""
        nd = self.nd
        capi.check(self.g.lib.parm_get_atoms(self.g.h, capi.dptr(self.out.numpy()), self.g.stride, 31))
        if not self.mixed:
            r = self.out
            return {"x": r[:, :nd], "v": r[:, nd:2 * nd], "a": r[:, 2 * nd:3 * nd], "f": r[:, 3 * nd:4 * nd]}
        r = self.out.to("cuda")
        return {"dx": (r[:, :nd] - self.x0).float(), "v": r[:, nd:2 * nd].float(), "a": r[:, 2 * nd:3 * nd].float(),
                "f": r[:, 3 * nd:4 * nd].float()}


def prepare(case, seed):
    return _State(case, seed)


def run(s):
    c, g = s.c, s.g
    if c["kind"] == "verlet":
        g.verlet(c["dt"], c["steps"])
        return s.records()
    if c["kind"] == "langevin":
        g.sol(c["dt"], DAMPING, 1.0, s.seed, c["steps"])
        return s.records()
    if c["kind"] == "damped":
        s.upload(s.frames[0])
        g.nlist_update(True)
        g.set_forces(True)
        g.damped(c["dt"], DAMPING, c["steps"])
        return s.records()
    if c["kind"] == "cg":
        s.upload(s.frames[0])
        g.nlist_update(True)
        g.nlcg_set_state(np.zeros(len(capi.NLCG_STATE)))
        g.nlcg_reset()
        g.nlcg_timestep(c["steps"])
        out = s.records()
        out["state"] = _shown(s, g.nlcg_state())
        return out
    s.upload(s.frames[s.turn % 2])
    s.turn += 1
    g.nlist_update(False)
    g.set_forces(True)
    e = {"energy": g.energy(), "virial": g.virial(), "stress": g.stress()}
    out = {k: _shown(s, v) for k, v in e.items()}
    out["contacts"], out["pairs"] = g.contacts().astype(np.int64), g.numpairs().astype(np.int64)
    f = s.records()
    out["f"], out["a"] = f["f"], f["a"]
    return out


def _shown(s, v):
    return v.astype(np.float32) if s.mixed else v


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _counts(c):
    """atoms, dimensions, interacting pairs (each once)."""
    if c["kind"] in ("verlet", "analyse"):
        n = c["nx"] * c["ny"] * c["nz"]
        return n, 3, 0.5 * n * (0.8 / SIGP ** 3) * 4.0 / 3.0 * math.pi * CUT ** 3
    srng = np.random.default_rng([c["nsys"], c["nmin"], c["nmax"]])
    n = int(np.exp(srng.uniform(np.log(c["nmin"]), np.log(c["nmax"] + 0.5), size=c["nsys"])).astype(int).sum())
    if c["kind"] == "langevin":
        return n, 3, 0.5 * n * (0.7 / SIGP ** 3) * 4.0 / 3.0 * math.pi
    return n, c["nd"], 0.5 * n * (6.0 if c["nd"] == 3 else 4.0)


def work(case):
    """Per step x and v read and written, the force written and read, 4 bytes and ~45 operations per pair; plus the
    records that cross the host link.  A minimiser step evaluates forces about five times."""
    n, nd, pairs = _counts(case)
    fb = 8 if case["prec"] == "fp64" else 4
    rec = 8.0 * n * (4 * nd + 1)
    step_bytes = n * nd * (32.0 + 2 * fb) + 4.0 * pairs
    if case["kind"] == "analyse":
        return {"bytes": 2 * rec + 5 * 4.0 * pairs + 4.0 * n * nd * 8, "flops": 5 * 45.0 * pairs}
    evals = case["steps"] * (5 if case["kind"] == "cg" else 1)
    links = 1 if case["kind"] in ("verlet", "langevin") else 2
    noise = 300.0 * n * evals if case["kind"] == "langevin" else 0.0
    return {"bytes": links * rec + evals * step_bytes, "flops": evals * 45.0 * pairs + noise}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch: the reference's algorithm (half list with its skin, rebuilt when the two largest
# displacements since the last build reach the skin)
# ---------------------------------------------------------------------------
class _Model:
    def __init__(self, c, seed):
        sizes, self.nd, L, x, v, self.kind, prm, self.skin = _inputs(c, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.sizes, self.off = sizes, np.concatenate([[0], np.cumsum(sizes)])
        self.Ls = torch.as_tensor(L, device=dev)
        self.sys = torch.repeat_interleave(torch.arange(len(sizes), device=dev), torch.as_tensor(sizes, device=dev))
        self.x, self.v, p = (torch.as_tensor(t, device=dev) for t in (x, v, prm))
        self.sig, self.third, self.dev = p[:, 1], float(prm[0, 2]), dev
        self.diam = self.sig * (self.third if self.kind == capi.LJCUT else 1.0)
        self.at = None
        self.f = torch.zeros_like(self.x)

    def image(self, d, s):
        L = self.Ls[s]
        return d - L * torch.round(d / L)

    def near(self, s):
        """pairs i < j of system s closer than its list thresholds."""
        lo, hi = int(self.off[s]), int(self.off[s + 1])
        x, L, nd = self.x[lo:hi], self.Ls[s], self.nd
        diam = self.diam[lo:hi]
        rmax = float(diam.max()) + self.skin
        nc = [int(k) for k in torch.floor(L / (rmax * (1 + 1e-9))).tolist()]
        n = hi - lo
        got = []

        def keep(i, j):
            d = x[i] - x[j]
            d = d - L * torch.round(d / L)
            ok = d.square().sum(-1).sqrt() < (diam[i] + diam[j]) / 2 + self.skin
            got.append((i[ok], j[ok]))

        if n < 3000 or min(nc) < 3:
            step = max(1, (1 << 24) // n)
            for a in range(0, n, step):
                i, j = torch.meshgrid(torch.arange(a, min(n, a + step), device=self.dev),
                                      torch.arange(n, device=self.dev), indexing="ij")
                up = i < j
                keep(i[up], j[up])
        else:
            fr = x / L
            nct = torch.tensor(nc, device=self.dev)
            ci = torch.minimum(((fr - fr.floor()) * nct).long(), nct - 1)
            cell = ci[:, 0]
            for d in range(1, nd):
                cell = cell * nc[d] + ci[:, d]
            ncell = int(np.prod(nc))
            cnt = torch.bincount(cell, minlength=ncell)
            start = torch.cumsum(cnt, 0) - cnt
            order = torch.argsort(cell)
            cap = int(cnt.max())
            table = torch.full((ncell, cap), -1, device=self.dev)
            table[cell[order], torch.arange(n, device=self.dev) - start[cell[order]]] = order
            rows = max(1, (1 << 23) // (cap * cap))
            for o in itertools.product((-1, 0, 1), repeat=nd):
                if o < (0,) * nd:
                    continue
                other = torch.roll(table.view(*nc, cap), [-k for k in o], list(range(nd))).reshape(ncell, cap)
                for a in range(0, ncell, rows):
                    i = table[a:a + rows, :, None].expand(-1, -1, cap)
                    j = other[a:a + rows, None, :].expand(-1, cap, -1)
                    ok = (i >= 0) & (j >= 0)
                    if not any(o):
                        ok &= i < j
                    keep(i[ok], j[ok])
        return torch.cat([g[0] for g in got]) + lo, torch.cat([g[1] for g in got]) + lo

    def rebuild(self):
        both = [self.near(s) for s in range(len(self.sizes))]
        self.i, self.j = (torch.cat([b[k] for b in both]) for k in (0, 1))
        self.at = self.x.clone()

    def trackers(self):
        """the displacement test, system by system (a rebuild of the others changes nothing that is summed)."""
        d = (self.x - self.at).square().sum(-1).sqrt()
        for s in range(len(self.sizes)):
            t = torch.topk(d[int(self.off[s]):int(self.off[s + 1])], 2).values
            if float(t.sum()) >= self.skin:
                self.rebuild()
                return

    def pairs(self):
        """displacement, its square, force scale and energy of every listed pair."""
        r = self.image(self.x[self.i] - self.x[self.j], self.sys[self.i])
        q = r.square().sum(-1)
        sg = (self.sig[self.i] + self.sig[self.j]) / 2
        zero = torch.zeros_like(q)
        if self.kind == capi.REPULSION:
            R = q.sqrt()
            b = (1 - R / sg).clamp(min=0.0)
            return r, torch.where(q > sg * sg, zero, b ** (self.third - 1) / sg / R), \
                torch.where(q > sg * sg, zero, b ** self.third / self.third)
        rs = q / (sg * sg)
        six = rs ** 3
        lj = self.kind == capi.LJCUT
        out = rs > (self.third ** 2 if lj else 1.0)
        shift = (1 - self.third ** -6) ** 2 if lj else 0.0
        return r, torch.where(out, zero, 12 / six * (1 / six - 1) / q), torch.where(out, zero, (1 - 1 / six) ** 2 - shift)

    def forces(self):
        r, s, _ = self.pairs()
        F = r * s[:, None]
        self.f = torch.zeros_like(self.x).index_add_(0, self.i, F).index_add_(0, self.j, -F)
        return self.f

    def by_system(self, t, s=None):
        return torch.zeros((len(self.sizes),) + t.shape[1:], dtype=t.dtype, device=self.dev).index_add_(
            0, self.sys if s is None else s, t)


def _philox_normals(key, step, n, dev):
    """Philox4x32-10 (Salmon et al. 2011) keyed per atom's system, Box-Muller: six normals for each atom of one system."""
    M = 0xFFFFFFFF
    out = []
    for blk in range(3):
        c = [torch.arange(n, device=dev), torch.full((n,), step & M, device=dev),
             torch.full((n,), (step >> 32) & M, device=dev), torch.full((n,), blk, device=dev)]
        k0, k1 = key & M, key >> 32

        def mul(a, b):   # 32 x 32 -> (hi, lo) in int64
            lo16, hi16 = b & 0xFFFF, b >> 16
            t = lo16 * a
            u = hi16 * a + (t >> 16)
            return u >> 16, ((u & 0xFFFF) << 16) | (t & 0xFFFF)
        for _ in range(10):
            h0, l0 = mul(0xD2511F53, c[0])
            h1, l1 = mul(0xCD9E8D57, c[2])
            c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M

        def unit(a, b):
            return (((a >> 5) << 26 | (b >> 6)).double() + 0.5) / 9007199254740992.0
        u1, u2 = unit(c[0], c[1]), unit(c[2], c[3])
        r = torch.sqrt(-2.0 * torch.log(u1))
        out += [r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2)]
    return torch.stack(out, 1)


def _splitmix(x):
    M = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & M
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & M
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & M
    return x ^ (x >> 31)


def _cg(m, steps):
    """CollectionNLCGV::reset and `steps` of its timestep (secant line search, Polak-Ribiere), every system its own."""
    dt, secmax, seceps, kmax = CG[0], CG[4], CG[5], CG[3]
    dot = lambda a, b: m.by_system((a * b).sum(-1))  # noqa: E731
    z = torch.zeros(len(m.sizes), dtype=torch.float64, device=m.dev)
    G = {k: z.clone() for k in capi.NLCG_STATE}
    m.a = m.v = m.forces().clone()
    for _ in range(steps):
        x = m.x
        m.x = x + m.v * dt
        eta0 = -dot(m.forces(), m.v)
        m.x = m.x + m.v * -dt
        m.trackers()
        m.forces()
        vdv = dot(m.v, m.v)
        G["alpha"], G["dxsum"], G["sec"] = z - dt, z.clone(), z.clone()
        loop = torch.ones_like(z, dtype=torch.bool)
        for _ in range(int(secmax)):
            if not bool(loop.any()):
                break
            eta = -dot(m.f, m.v)
            fac = -eta / (eta0 - eta).abs()
            flat = (eta0 - eta).abs() <= 1e-12 * eta.abs()
            fac = torch.where(flat, 1.1, fac)
            sec = torch.where(flat, torch.where(G["sec"] > 0, G["sec"] * 2 - 1, 1.0), G["sec"])
            alpha = G["alpha"].abs() * fac
            G["alpha"], G["sec"] = torch.where(loop, alpha, G["alpha"]), torch.where(loop, sec, G["sec"])
            G["dxsum"] = torch.where(loop, G["dxsum"] + alpha, G["dxsum"])
            m.x = torch.where(loop[m.sys][:, None], m.x + m.v * alpha[m.sys][:, None], m.x)
            m.trackers()
            m.forces()
            eta0 = torch.where(loop, eta, eta0)
            done = G["alpha"] ** 2 * vdv < seceps ** 2
            G["sec"] = torch.where(loop & ~done, G["sec"] + 1, G["sec"])
            loop = loop & ~done & (G["sec"] < secmax)
        G["alphavmax"] = (G["alpha"] ** 2 * vdv).sqrt()
        old, mid = G["Knew"], dot(m.f, m.a)
        G["Knew"] = dot(m.f, m.f)
        G["beta"] = (G["Knew"] - mid) / old
        G["k"] = G["k"] + 1
        b = G["beta"]
        restart = (G["k"] >= kmax) | ~torch.isfinite(b) | (b <= 0)
        G["k"] = torch.where(restart, 0.0, G["k"])
        G["betaused"] = torch.where(restart, 0.0, b.clamp(max=1.0))
        m.a = m.f.clone()
        m.v = m.a + m.v * G["betaused"][m.sys][:, None]
    return torch.stack([G[k] for k in capi.NLCG_STATE], 1)


def exact(case, seed):
    c = case
    m = _Model(c, seed)
    m.rebuild()
    x0 = m.x
    out = {}
    if c["kind"] == "analyse":
        r, s, e = m.pairs()
        at = m.sys[m.i]
        rf = r[:, :, None] * (r * s[:, None])[:, None, :]
        f = m.forces()
        return {"energy": m.by_system(e, at), "virial": m.by_system((r * r).sum(-1) * s, at),
                "stress": m.by_system(rf, at), "contacts": None, "pairs": None, "f": f, "a": f}
    if c["kind"] == "cg":
        out["state"] = _cg(m, c["steps"])
        a = m.a
    else:
        a = m.forces()
        dt = c["dt"]
        h = DAMPING * dt
        c0, c1 = math.exp(-h), -math.expm1(-h) / h
        c2 = (1 - c1) / h
        if c["kind"] == "verlet":
            c0, c1, c2 = 1.0, 1.0, 0.5
        # BivariateGauss::set: deviations of the position and velocity noise and their correlation
        sr = math.sqrt((1 / h) * (2 - (-4 * math.expm1(-h) + math.expm1(-2 * h)) / h)) if h > 1e-4 else 0.0
        sv = math.sqrt(-math.expm1(-2 * h))
        corr = math.expm1(-h) ** 2 / h / sr / sv if sr else 0.0
        for k in range(c["steps"]):
            m.x = m.x + (m.v * (c1 * dt) + a * (c2 * dt * dt))
            m.v = m.v * c0 + a * (dt * (c1 - c2))
            if c["kind"] == "langevin":
                g = torch.cat([_philox_normals(_splitmix(int(seed) + s), k + 1, n, m.dev)
                               for s, n in enumerate(m.sizes)])
                m.x = m.x + g[:, :3] * (sr * dt)
                m.v = m.v + (g[:, :3] * (sv * corr) + g[:, 3:] * (sv * math.sqrt(1 - corr * corr)))
            a = m.forces()
            m.v = m.v + a * (dt * c2)
            m.trackers()
    if c["prec"] == "mixed":
        out["dx"] = m.x - x0
    else:
        out["x"] = m.x
    out.update(v=m.v, a=a, f=m.f)
    return out
