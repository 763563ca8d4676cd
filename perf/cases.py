"""The work a user of this framework gives it, as measurable cases.

Two kinds of system:

* ``chain``: the seeded lattice chain of geodesic_cuda.synth as a droplet in
  vacuum (non-periodic, Lennard-Jones, Coulomb, scaled 1-4 pairs, bonds,
  angles, dihedrals), the system of the benchmark's configurations.  One
  pre-relaxed droplet per size; a seed gives it its own rigid rotation and
  Maxwell-Boltzmann velocities.
* ``water``: a periodic box of three-site water at 0.1 atoms per cubic
  Angstrom, a lattice of columns with alternating dipoles, each molecule
  displaced and turned a little by the seed.

Each case is driven through `geodesic_cuda.backend.CudaBackend`, the way the
run loop or a host engine drives it:

* ``steps``: `steps()`, a block of BAB steps on host arrays, state in place;
* ``forces``: `compute_forces()` on positions moved within the skin;
* ``build``: `build_neighbor_list()` and `compute_forces()`, new positions;
* ``trait``: one step through the trait's methods, one call each;
* ``resident``: a batch of systems advanced on the device, its energies and
  its state read back;
* ``frames``: resident steps that record trajectory frames, taken once.

Steps continue the trajectory of the pass before, as a run does.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodesic-m_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from geodesic_cuda import amber, backend, synth  # noqa: E402

RC, RLIST, RSW = 10.0, 12.0, 8.0  # cutoff, list radius, switch radius of the benchmark's systems
KC = 332.0522173
ACC = 20.455 * 20.455
MAX_ITER, TOL = 200, 1e-10
KB = 0.0019872041  # kcal/mol/K


def listed():
    return [
        # the smallest: a peptide-sized molecule in vacuum, where launches and latency count
        dict(name="chain_224_steps", kind="steps", system="chain", n=224, fp64=False, constrained=False, steps=50),
        # a small periodic box with constrained O-H bonds, a short run
        dict(name="water_1536_constrained", kind="steps", system="water", n=1536, fp64=False, constrained=True, steps=20),
        # the reference-precision run of 5,000 atoms
        dict(name="chain_5000_fp64", kind="steps", system="chain", n=5000, fp64=True, constrained=False, steps=5),
        # the headline system, one step per call from a host engine
        dict(name="chain_50000_one_step", kind="steps", system="chain", n=50000, fp64=False, constrained=False, steps=1),
        # a chain with 40 % hydrogens, their bonds constrained
        dict(name="chain_20011_constrained", kind="steps", system="chain", n=20011, fp64=False, constrained=True, steps=5),
        # an ordinary solvated-box size, flexible bonds, a block of steps
        dict(name="water_98304_steps", kind="steps", system="water", n=98304, fp64=False, constrained=False, steps=10),
        # FP64 forces of a periodic box (an engine that keeps its own integrator)
        dict(name="water_12000_fp64_forces", kind="forces", system="water", n=12000, fp64=True, constrained=False, steps=1),
        # a list build and a force evaluation on new positions
        dict(name="water_46875_build", kind="build", system="water", n=46875, fp64=False, constrained=False, steps=1),
        # one step of the run loop through the trait's methods
        dict(name="water_5184_trait", kind="trait", system="water", n=5184, fp64=False, constrained=True, steps=1),
        # a batch of uneven small systems (replicas, ligands)
        dict(name="chains_24_resident", kind="resident", system="chain", n=1500, fp64=False, constrained=False, steps=10, systems=24),
        # a run with trajectory output
        dict(name="water_24000_frames", kind="frames", system="water", n=24000, fp64=False, constrained=True, steps=10),
        # the largest: a virus-sized box
        dict(name="water_786432_steps", kind="steps", system="water", n=786432, fp64=False, constrained=False, steps=3),
    ]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["steps", "steps", "steps", "forces", "build", "trait", "resident", "frames"])
    fp64 = rng.random() < 0.25
    system = "chain" if kind == "resident" else rng.choice(["chain", "water"])
    constrained = kind in ("trait", "frames") or (kind == "steps" and rng.random() < 0.4)
    if kind == "resident":
        return dict(kind=kind, system=system, n=int(math.exp(rng.uniform(math.log(300), math.log(2500)))), fp64=fp64,
                    constrained=False, steps=rng.randint(2, 20), systems=rng.randint(3, 32))
    hi = 40000 if system == "chain" else 400000
    if fp64 or kind != "steps":
        hi = min(hi, 60000)
    n = int(math.exp(rng.uniform(math.log(150), math.log(hi))))
    if system == "water":
        n = max(n // 3 * 3, 192)
    elif n < 1500:
        n = max(n // 32 * 32, 160)
    most = 50 if n < 10000 else 20 if n < 60000 else 5
    if kind in ("forces", "build", "trait"):
        steps = 1
    elif kind == "frames":
        steps = 2 * rng.randint(1, 10)
    else:
        steps = rng.randint(1, max(1, most // 4 if fp64 else most))
    return dict(kind=kind, system=system, n=n, fp64=fp64, constrained=constrained, steps=steps)


# ---------------------------------------------------------------- systems

_chains = {}


def _chain(n, h_fraction, which):
    """A pre-relaxed droplet (one per size), with H bonds as constraints when it has hydrogens."""
    key = (n, h_fraction, which)
    if key not in _chains:
        if len(_chains) > 64:
            _chains.clear()
        iters = int(min(200, max(40, 2.5e6 / n)))
        atoms, topo, state, _ = synth.generate(n, seed=1009 + which, h_fraction=h_fraction, temperature=300.0, relax_iters=iters)
        if h_fraction > 0:
            topo = amber.promote_hydrogen_bonds(topo, atoms)
        _chains[key] = (atoms, topo, np.ascontiguousarray(state.pos))
    return _chains[key]


def _rotation(r):
    q, t = np.linalg.qr(r.standard_normal((3, 3)))
    q = q * np.sign(np.diag(t))
    return q if np.linalg.det(q) > 0 else -q


def _velocities(mass, r, temperature=300.0):
    v = r.standard_normal((3, len(mass))) * np.sqrt(KB * temperature * ACC / mass)
    return v - (v * mass).sum(axis=1, keepdims=True) / mass.sum()


def _chain_system(case, seed, which=0):
    atoms, topo, base = _chain(case["n"], 0.4 if case["constrained"] else 0.0, which)
    r = np.random.default_rng([seed, which, 17])
    c = base.mean(axis=1, keepdims=True)
    pos = np.ascontiguousarray(_rotation(r) @ (base - c) + c)
    return atoms, topo, pos, np.ascontiguousarray(_velocities(atoms.mass, r))


def _water_box(n):
    """Cells along x, y, z (even in x and y, where the columns alternate, when that can be) and the box."""
    m = n // 3
    best = None
    side = m ** (1.0 / 3.0)
    for a in range(max(2, int(side * 0.6)), int(side * 1.5) + 2):
        for b in range(a, int(side * 1.7) + 2):
            c = -(-m // (a * b))
            if c < 2:
                continue
            score = (a * b * c - m) / m + 0.02 * (a % 2 + b % 2) + 0.1 * (max(a, b, c) / min(a, b, c) - 1)
            if best is None or score < best[0]:
                best = (score, a, b, c)
    _, a, b, c = best
    edge = (m / 0.1 * 3.0 / (a * b * c)) ** (1.0 / 3.0)
    return a, b, c, edge


def _water_system(case, seed):
    n = case["n"] // 3 * 3
    m = n // 3
    a, b, c, edge = _water_box(n)
    r = np.random.default_rng([seed, 23])
    k = np.arange(m) if a * b * c == m else np.sort(r.permutation(a * b * c)[:m])
    ix, iy, iz = k % a, (k // a) % b, k // (a * b)
    o = (np.stack([ix, iy, iz]) + 0.5) * edge + r.uniform(-0.08, 0.08, (3, m))
    sign = np.where((ix + iy) % 2 == 0, 1.0, -1.0)
    half, d = math.radians(104.52 / 2), 0.9572
    phi = r.normal(0.25 * math.pi, 0.15, m)
    ex = np.stack([np.cos(phi), np.sin(phi), r.normal(0, 0.1, m)])
    ez = np.stack([r.normal(0, 0.1, m), r.normal(0, 0.1, m), sign])
    ez /= np.linalg.norm(ez, axis=0)
    ex -= ez * (ex * ez).sum(axis=0)
    ex /= np.linalg.norm(ex, axis=0)
    pos = np.empty((3, m, 3))
    pos[:, :, 0] = o
    pos[:, :, 1] = o + d * (math.cos(half) * ez + math.sin(half) * ex)
    pos[:, :, 2] = o + d * (math.cos(half) * ez - math.sin(half) * ex)
    box = np.array([a * edge, b * edge, c * edge])
    pos = np.ascontiguousarray(pos.reshape(3, n))
    pos = pos - box[:, None] * np.floor(pos / box[:, None])
    rep = lambda v, t: np.tile(np.array(v, dtype=t), m)  # noqa: E731
    i0 = (3 * np.arange(m)).astype(np.uint32)
    pair = lambda u, v: (np.stack([i0 + np.uint32(x) for x in u], 1).reshape(-1), np.stack([i0 + np.uint32(x) for x in v], 1).reshape(-1))  # noqa: E731
    atoms = amber.AtomData(rep([3.1507, 0.4, 0.4], np.float64), rep([0.1521, 0.046, 0.046], np.float64),
                           rep([15.9994, 1.008, 1.008], np.float64), rep([-0.834, 0.417, 0.417], np.float64),
                           rep([3, 0, 0], np.uint8), np.zeros(n, np.uint32), [])
    topo = amber.BondedTopology.empty()
    bi, bj = pair([0, 0], [1, 2])
    if case["constrained"]:
        topo.constr_i, topo.constr_j, topo.constr_dsq = bi, bj, np.full(2 * m, d * d)
    else:
        topo.bond_i, topo.bond_j, topo.bond_k, topo.bond_r0 = bi, bj, np.full(2 * m, 450.0), np.full(2 * m, d)
    topo.angle_i, topo.angle_j, topo.angle_k = i0 + np.uint32(1), i0, i0 + np.uint32(2)
    topo.angle_kth, topo.angle_th0 = np.full(m, 55.0), np.full(m, 2 * half)
    topo.excl_i, topo.excl_j = pair([0, 0, 1], [1, 2, 2])
    return atoms, topo, np.ascontiguousarray(pos), np.ascontiguousarray(_velocities(atoms.mass, r, 400.0)), box


def _params(case, box):
    water = case["system"] == "water"
    # a box smaller than two list radii takes shorter radii, as a user's would
    scale = min(1.0, 0.499 * min(box) / RLIST) if water else 1.0
    return backend.SimParams(box_size=tuple(float(x) for x in box), periodic=water, r_cutoff=RC * scale,
                             r_skin=RLIST * scale, r_switch=RSW * scale, coulomb=True, scale14_lj=0.0 if water else 0.5,
                             scale14_coul=0.0 if water else 1.0 / 1.2, max_constr_iter=MAX_ITER, constr_tol=TOL,
                             precision=backend.PRECISION_FP64 if case["fp64"] else backend.PRECISION_MIXED,
                             bonded_min_image=water)


def _inputs(case, seed):
    if case["system"] == "water":
        atoms, topo, pos, vel, box = _water_system(case, seed)
        return atoms, topo, pos, vel, _params(case, box)
    atoms, topo, pos, vel = _chain_system(case, seed)
    return atoms, topo, pos, vel, _params(case, (10000.0,) * 3)


def _dt(case):
    """2 fs; 1 fs where water's O-H bonds are flexible."""
    return 0.001 if case["system"] == "water" and not case["constrained"] else 0.002


def _batch_sizes(case):
    """Uneven systems, the largest 16 times the smallest, the largest first."""
    k = case["systems"]
    return [max(60, int(case["n"] * 4.0 ** (1.0 - 2.0 * i / max(k - 1, 1)))) for i in range(k)]


def _moved(pos, seed):
    """Positions a fraction of the skin away from the list's, as between two rebuilds."""
    return np.ascontiguousarray(pos + np.random.default_rng([seed, 31]).uniform(-0.05, 0.05, pos.shape))


def _pinned(a):
    """A host array in pinned memory, as an engine keeps the arrays it exchanges every step."""
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    v = t.numpy()
    v[...] = a
    return v


def prepare(case, seed):
    if case["kind"] == "resident":
        systems = [_chain_system(dict(case, n=n), seed, which) for which, n in enumerate(_batch_sizes(case))]
        be = backend.CudaBackend.ensemble([s[0] for s in systems], [s[1] for s in systems], _params(case, (10000.0,) * 3))
        pos = np.ascontiguousarray(np.concatenate([s[2] for s in systems], axis=1))
        vel = np.ascontiguousarray(np.concatenate([s[3] for s in systems], axis=1))
        be.upload_state(pos, vel)
        be.forces_resident()
        return dict(case=case, be=be, pos=pos, vel=vel, dt=_dt(case))
    atoms, topo, pos, vel, params = _inputs(case, seed)
    be = backend.CudaBackend(atoms, topo, params)
    state = dict(case=case, be=be, dt=_dt(case))
    if case["kind"] == "build":
        state["pos"] = pos
        return state
    pos, vel = _pinned(pos), _pinned(vel)
    be.build_neighbor_list(pos)
    if case["constrained"]:
        be.constrain_velocities(pos, vel)
    if case["kind"] == "forces":
        pos = _moved(pos, seed)
    if case["kind"] == "frames":
        be.frames_enable(2, case["steps"] // 2)
        be.upload_state(pos, vel)
    if case["kind"] == "trait":
        state["forces"] = be.compute_forces(pos)
    state.update(pos=pos, vel=vel)
    return state


def run(state):
    case, be, pos, dt = state["case"], state["be"], state["pos"], state["dt"]
    kind = case["kind"]
    if kind == "steps":
        energy, _, _ = be.steps(pos, state["vel"], dt, case["steps"])
        return {"pos": pos, "vel": state["vel"], "energy": energy}
    if kind == "forces":
        return {"forces": be.compute_forces(pos), "energy": be.potential_energy()}
    if kind == "build":
        be.build_neighbor_list(pos)
        return {"pos": pos, "forces": be.compute_forces(pos), "energy": be.potential_energy()}
    if kind == "trait":
        vel = state["vel"]
        be.half_kick(vel, state["forces"], dt / 2)
        be.geodesic_drift(pos, vel, dt)
        if be.needs_rebuild(pos):
            be.build_neighbor_list(pos)
        state["forces"] = be.compute_forces(pos)
        be.half_kick(vel, state["forces"], dt / 2)
        be.constrain_velocities(pos, vel)
        return {"pos": pos, "vel": vel, "forces": state["forces"], "energy": be.potential_energy(), "kinetic": be.kinetic_energy(vel)}
    be.run_resident(dt, case["steps"])
    if kind == "frames":
        f = be.frames_take()
        return {"xyz": f["xyz"], "e_pot": f["e_pot"], "e_kin": f["e_kin"]}
    e_pot, e_kin = be.ensemble_energies()
    be.download_state(pos, state["vel"])
    return {"pos": pos, "vel": state["vel"], "e_pot": e_pot, "e_kin": e_kin}


def work(case):
    """Per force evaluation: 4 B per pair of the half list and 52 B per atom (positions, parameters, forces), and about
    50 operations per pair within the cutoff; per step 248 B per atom of integrator state; a build writes the list."""
    n = case["n"] if case["kind"] != "resident" else sum(_batch_sizes(case))
    scale = 1.0
    if case["system"] == "water":
        scale = min(1.0, 0.499 * min(_water_box(n)[k] for k in range(3)) * _water_box(n)[3] / RLIST)
    inside = lambda r: min(4.0 / 3.0 * math.pi * (r * scale) ** 3 * 0.1, n if case["kind"] != "resident" else case["n"])  # noqa: E731
    listed_pairs, pairs = n * inside(RLIST) / 2, n * inside(RC) / 2
    per_eval = 4 * listed_pairs + 52 * n
    if case["kind"] == "build":
        return {"bytes": per_eval + 4 * listed_pairs + 44 * n, "flops": 50 * pairs + 8 * listed_pairs}
    if case["kind"] == "forces":
        return {"bytes": per_eval, "flops": 50 * pairs}
    return {"bytes": case["steps"] * (per_eval + 248 * n), "flops": case["steps"] * (50 * pairs + 60 * n)}


# ---------------------------------------------- the same in 64 bits, in torch


class _Exact:
    """Forces, constraints and steps in FP64 with torch operations."""

    def __init__(self, atoms, topo, p):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        f = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)  # noqa: E731
        i = lambda a: torch.as_tensor(np.asarray(a).astype(np.int64), device=self.dev)  # noqa: E731
        self.p, self.t, self.n = p, topo, len(atoms.mass)
        self.sig, self.eps, self.q, self.mass = f(atoms.sigma), f(atoms.epsilon), f(atoms.charge), f(atoms.mass)
        self.inv_m = 1.0 / self.mass
        self.box = f(p.box_size)
        self.bonds = (i(topo.bond_i), i(topo.bond_j), f(topo.bond_k), f(topo.bond_r0))
        self.angles = (i(topo.angle_i), i(topo.angle_j), i(topo.angle_k), f(topo.angle_kth), f(topo.angle_th0))
        live = np.asarray(topo.dihed_kphi) != 0
        self.diheds = tuple(i(np.asarray(x)[live]) for x in (topo.dihed_i, topo.dihed_j, topo.dihed_k, topo.dihed_l)) + (
            f(np.asarray(topo.dihed_kphi)[live]), f(np.asarray(topo.dihed_n)[live]), f(np.asarray(topo.dihed_delta)[live]))
        self.constr = (i(topo.constr_i), i(topo.constr_j), f(topo.constr_dsq))
        key = lambda a, b: np.minimum(a, b).astype(np.int64) * self.n + np.maximum(a, b).astype(np.int64)  # noqa: E731
        self.excl = torch.as_tensor(np.unique(key(topo.excl_i, topo.excl_j)), device=self.dev)
        p14 = np.zeros(0, np.int64)
        if p.scale14_lj or p.scale14_coul:
            close = np.concatenate([key(topo.bond_i, topo.bond_j), key(topo.angle_i, topo.angle_k)])
            p14 = key(topo.dihed_i, topo.dihed_l)[np.asarray(topo.dihed_i) != np.asarray(topo.dihed_l)]
            p14 = np.setdiff1d(np.unique(p14), close)
        self.p14 = (i(p14 // self.n), i(p14 % self.n))
        self.list_pos = None

    def image(self, d):
        """Nearest image of the differences d (3, m)."""
        if not self.p.periodic:
            return d
        L = self.box[:, None]
        s = d / L
        return d - L * torch.sign(s) * torch.floor(s.abs() + 0.5)

    def pairs(self, x):
        """Pairs within the cutoff and a margin, kept until an atom has moved half the margin."""
        margin = 0.4
        if self.list_pos is not None and float(self.image(x - self.list_pos).square().sum(0).max()) < (margin / 2) ** 2:
            return self.pi, self.pj
        rl2, pi, pj = (self.p.r_cutoff + margin) ** 2, [], []
        rows = max(1, min(self.n, 40_000_000 // self.n))
        for a in range(0, self.n, rows):
            b = min(self.n, a + rows)
            r2 = torch.zeros((b - a, self.n - a), dtype=torch.float32, device=self.dev)
            for k in range(3):
                d = (x[k, a:b, None] - x[k, None, a:]).float()
                if self.p.periodic:
                    L = float(self.box[k])
                    d -= L * torch.round(d / L)
                r2 += d * d
            u, v = torch.nonzero(r2 <= rl2, as_tuple=True)
            keep = v > u
            pi.append(u[keep] + a)
            pj.append(v[keep] + a)
        pi, pj = torch.cat(pi), torch.cat(pj)
        if len(self.excl):
            keep = ~torch.isin(pi * self.n + pj, self.excl)
            pi, pj = pi[keep], pj[keep]
        self.pi, self.pj, self.list_pos = pi, pj, x.clone()
        return pi, pj

    def add(self, f, i, v):
        for k in range(3):
            f[k].index_add_(0, i, v[k])

    def pair_terms(self, x, f, i, j, switch, s_lj=1.0, s_q=1.0):
        energy = 0.0
        for a in range(0, len(i), 20_000_000):
            u, v = i[a:a + 20_000_000], j[a:a + 20_000_000]
            d = x[:, v] - x[:, u]
            d = self.image(d)
            r2 = (d * d).sum(0)
            if switch:
                keep = r2 <= self.p.r_cutoff ** 2
                u, v, d, r2 = u[keep], v[keep], d[:, keep], r2[keep]
            r = r2.sqrt()
            s6 = (0.5 * (self.sig[u] + self.sig[v]) / r) ** 6
            e4 = 4.0 * (self.eps[u] * self.eps[v]).sqrt() * s_lj
            vc = KC * self.q[u] * self.q[v] / r * s_q
            pot = e4 * s6 * (s6 - 1.0) + vc
            fr = (6.0 * e4 * s6 * (2.0 * s6 - 1.0) + vc) / r
            if switch:
                w = self.p.r_cutoff - self.p.r_switch
                y = ((r - self.p.r_switch) / w).clamp(min=0.0)
                sw = 1.0 - y ** 3 * (10.0 - 15.0 * y + 6.0 * y * y)
                fr = fr * sw + pot * 30.0 * y * y * (1.0 - y) ** 2 / w
                pot = pot * sw
            energy += float(pot.sum())
            g = d * (fr / r)
            self.add(f, u, -g)
            self.add(f, v, g)
        return energy

    def bonded(self, x):
        e = torch.zeros((), dtype=torch.float64, device=self.dev)
        i, j, k, r0 = self.bonds
        if len(i):
            e = e + (k * (self.image(x[:, j] - x[:, i]).square().sum(0).sqrt() - r0) ** 2).sum()
        i, j, kk, k, th0 = self.angles
        if len(i):
            a, b = self.image(x[:, i] - x[:, j]), self.image(x[:, kk] - x[:, j])
            c = (a * b).sum(0) / (a.square().sum(0) * b.square().sum(0)).sqrt()
            e = e + (k * (torch.acos(c) - th0) ** 2).sum()
        i, j, kk, m, k, mult, delta = self.diheds
        if len(i):
            b1, b2, b3 = self.image(x[:, j] - x[:, i]), self.image(x[:, kk] - x[:, j]), self.image(x[:, m] - x[:, kk])
            u, v = torch.linalg.cross(b1, b2, dim=0), torch.linalg.cross(b2, b3, dim=0)
            y = (torch.linalg.cross(u, v, dim=0) * b2).sum(0) / b2.square().sum(0).sqrt()
            e = e + (k * (1.0 + torch.cos(mult * torch.atan2(y, (u * v).sum(0)) - delta))).sum()
        return e

    def forces(self, x):
        xg = x.detach().clone().requires_grad_(True)
        e = self.bonded(xg)
        f = -torch.autograd.grad(e, xg)[0] if e.requires_grad else torch.zeros_like(x)
        e = float(e.detach())
        e += self.pair_terms(x, f, *self.p14, False, self.p.scale14_lj, self.p.scale14_coul) if len(self.p14[0]) else 0.0
        return f, e + self.pair_terms(x, f, *self.pairs(x), True)

    def shake(self, x, ref):
        i, j, dsq = self.constr
        r = self.image(ref[:, i] - ref[:, j])
        for _ in range(MAX_ITER):
            d = self.image(x[:, i] - x[:, j])
            lam = ((d * d).sum(0) - dsq) / (2.0 * (self.inv_m[i] + self.inv_m[j]) * (d * r).sum(0))
            self.add(x, i, -lam * self.inv_m[i] * r)
            self.add(x, j, lam * self.inv_m[j] * r)
            if float(lam.abs().max()) < TOL:
                return

    def rattle(self, x, v):
        i, j, _ = self.constr
        r = self.image(x[:, i] - x[:, j])
        w = (self.inv_m[i] + self.inv_m[j]) * (r * r).sum(0)
        for _ in range(MAX_ITER):
            mu = ((v[:, i] - v[:, j]) * r).sum(0) / w
            self.add(v, i, -mu * self.inv_m[i] * r)
            self.add(v, j, mu * self.inv_m[j] * r)
            if float(mu.abs().max()) < TOL:
                return

    def wrap(self, x):
        L = self.box[:, None]
        return x - L * torch.floor(x / L) if self.p.periodic else x

    def kinetic(self, v):
        return 0.5 * float((self.mass * (v * v).sum(0)).sum()) / ACC

    def step(self, x, v, f, dt):
        v = v + dt / 2 * ACC * f * self.inv_m
        ref = x.clone()
        x = x + dt * v
        if len(self.constr[0]):
            self.shake(x, ref)
        v = (x - ref) / dt
        return x, v

    def finish(self, x, v, f, dt):
        v = v + dt / 2 * ACC * f * self.inv_m
        if len(self.constr[0]):
            self.rattle(x, v)
        return v


def exact(case, seed):
    """A run's outputs in 64 bits.  A periodic step case returns no positions: the list rebuilds wrap atoms into the box
    at times that its list's skin decides."""
    kind = case["kind"]
    n = case["n"] if kind != "resident" else sum(_batch_sizes(case))
    if kind == "resident":
        parts = []
        for which, m in enumerate(_batch_sizes(case)):
            atoms, topo, pos, vel = _chain_system(dict(case, n=m), seed, which)
            parts.append(_exact_steps(case, _Exact(atoms, topo, _params(case, (10000.0,) * 3)), pos, vel))
        return {"pos": np.concatenate([q[0] for q in parts], 1), "vel": np.concatenate([q[1] for q in parts], 1),
                "e_pot": np.array([q[2] for q in parts]), "e_kin": np.array([q[3] for q in parts])}
    if n > 110_000 or (kind in ("steps", "frames") and n * (2 + case["steps"]) > 1_500_000):
        return None
    atoms, topo, pos, vel, p = _inputs(case, seed)
    ex = _Exact(atoms, topo, p)
    x = ex.wrap(torch.as_tensor(pos, device=ex.dev))
    if kind in ("forces", "build"):
        if kind == "forces":
            x = torch.as_tensor(_moved(x.cpu().numpy(), seed), device=ex.dev)
        f, e = ex.forces(x)
        out = {"forces": f.cpu().numpy(), "energy": e}
        return dict(out, pos=x.cpu().numpy()) if kind == "build" else out
    free = None if p.periodic else True
    if kind == "frames":
        x, v, f = _exact_start(case, ex, pos, vel)
        xyz, ep, ek = [], [], []
        for k in range(case["steps"]):
            x, v = ex.step(x, v, f, _dt(case))
            f, e = ex.forces(x)
            v = ex.finish(x, v, f, _dt(case))
            if k % 2 == 1:
                xyz.append(x.cpu().numpy())
                ep.append(e)
                ek.append(ex.kinetic(v))
        return {"xyz": free and np.stack(xyz), "e_pot": np.array(ep), "e_kin": np.array(ek)}
    x, v, e, ke, f = _exact_steps(case, ex, pos, vel)
    out = {"pos": free and x, "vel": v, "energy": e}
    return dict(out, forces=f, kinetic=ke) if kind == "trait" else out


def _exact_start(case, ex, pos, vel):
    x = ex.wrap(torch.as_tensor(pos, device=ex.dev)).clone()
    v = torch.as_tensor(vel, device=ex.dev).clone()
    if len(ex.constr[0]):
        ex.rattle(x, v)
    return x, v, ex.forces(x)[0]


def _exact_steps(case, ex, pos, vel):
    x, v, f = _exact_start(case, ex, pos, vel)
    e = 0.0
    for _ in range(case["steps"]):
        x, v = ex.step(x, v, f, _dt(case))
        f, e = ex.forces(x)
        v = ex.finish(x, v, f, _dt(case))
    return x.cpu().numpy(), v.cpu().numpy(), e, ex.kinetic(v), f.cpu().numpy()
