"""The performance cases of the femmd2D timestep: what a user's program has
this framework do, from one small run to the largest single-GPU system.

Every pass starts from given positions and velocities (page-locked host
buffers, as a program that feeds and stores states keeps them), makes the
calls of the public entry points, and reads the results back:

  run      set_state, run(steps), get_state, energies: the reference's run
           loop.  LJ fluids in both force modes (the reference-exact one is the
           default), elastomer suspensions, and disks in solvent.
  forces   set_state, build_nn, calc_forces, forces and particle energies: one
           evaluation, as an external integrator or minimiser asks for it.  A
           two-kind fluid whose sizes vary from particle to particle.
  batch    independent replicas of uneven sizes through Batch.run.
  adjoint  adjoint_forward, the observable and adjoint_backward of disks
           compressed by a moving wall: one iteration of a fit.

Sizes come from the benchmark's workloads (4096 atoms, 256 disks, 4096 disks
in 1,000,000 solvent particles, the replica ensemble, 64 compressed disks) and
from the range between them, odd ones among them.  All inputs are synthetic
and made from the seed alone.
"""
import math

import numpy as np
import torch

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S

MODES = {"reference": 0, "fast": 1}
MAX_RUN_ATOM_STEPS = 80e6  # of the largest listed run: 1,520,192 atoms, 50 steps


def listed():
    return [
        # the smallest calls: latency and launches count
        {"name": "lj_400_reference_run20", "kind": "run", "system": "lj", "mode": "reference", "side": 20,
         "density": 0.8, "T": 1.0, "steps": 20},
        # the benchmark's small fluid in the mode it is run in
        {"name": "lj_4096_fast_run100", "kind": "run", "system": "lj", "mode": "fast", "side": 64, "density": 0.8,
         "T": 1.0, "steps": 100},
        # an odd size in the default mode
        {"name": "lj_10201_reference_run50", "kind": "run", "system": "lj", "mode": "reference", "side": 101,
         "density": 0.7, "T": 1.2, "steps": 50},
        # an ordinary and the largest fluid in the fast mode
        {"name": "lj_90000_fast_run50", "kind": "run", "system": "lj", "mode": "fast", "side": 300, "density": 0.8,
         "T": 1.0, "steps": 50},
        {"name": "lj_1m_fast_run50", "kind": "run", "system": "lj", "mode": "fast", "side": 1000, "density": 0.8,
         "T": 1.0, "steps": 50},
        # the benchmark's elastomer suspension: bonds, triangles, contacts
        {"name": "suspension_256_run100", "kind": "run", "system": "suspension", "mode": "reference", "side": 16,
         "steps": 100},
        # disks in solvent: an ordinary size in the fast mode, the largest in the default mode
        {"name": "mixed_144_50k_fast_run50", "kind": "run", "system": "mixed", "mode": "fast", "side": 12,
         "solvent": 50000, "steps": 50},
        {"name": "mixed_4096_1m_run50", "kind": "run", "system": "mixed", "mode": "reference", "side": 64,
         "solvent": 1000000, "steps": 50},
        # one evaluation of a two-kind fluid with a size per particle
        {"name": "forces_30976_polydisperse", "kind": "forces", "mode": "reference", "side": 176, "density": 0.75},
        # fewer replicas than the card has SMs, sizes log-uniform as the benchmark's ensemble
        {"name": "batch_128_run100", "kind": "batch", "replicas": 128, "n_min": 500, "n_max": 20000, "steps": 100},
        # forward and backward: the benchmark's differentiable compression
        {"name": "adjoint_64_200_every20", "kind": "adjoint", "side": 8, "steps": 200, "every": 20},
    ]


def _log_uniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["lj", "lj", "lj", "suspension", "mixed", "mixed", "forces", "batch", "adjoint"])
    if kind == "lj":
        side = round(_log_uniform(rng, 17, 1000))
        steps = min(rng.randint(10, 100), int(MAX_RUN_ATOM_STEPS * 0.6 / side ** 2))
        return {"kind": "run", "system": "lj", "mode": rng.choice(["fast", "reference"]), "side": side,
                "density": round(rng.uniform(0.6, 0.85), 3), "T": round(rng.uniform(0.5, 1.5), 2), "steps": steps}
    if kind == "suspension":
        return {"kind": "run", "system": "suspension", "mode": rng.choice(["fast", "reference"]),
                "side": round(_log_uniform(rng, 2, 40)), "steps": rng.randint(10, 100)}
    if kind == "mixed":
        side = round(_log_uniform(rng, 4, 40))
        return {"kind": "run", "system": "mixed", "mode": rng.choice(["fast", "reference"]), "side": side,
                "solvent": round(side * side * rng.uniform(220, 500)), "steps": rng.randint(10, 60)}
    if kind == "forces":
        return {"kind": "forces", "mode": rng.choice(["fast", "reference"]), "side": round(_log_uniform(rng, 18, 600)),
                "density": round(rng.uniform(0.6, 0.8), 3)}
    if kind == "batch":
        return {"kind": "batch", "replicas": round(_log_uniform(rng, 6, 128)), "n_min": 500,
                "n_max": round(_log_uniform(rng, 2000, 20000)), "steps": rng.randint(20, 100)}
    return {"kind": "adjoint", "side": rng.randint(2, 8), "steps": rng.randint(40, 200), "every": rng.randint(10, 40)}


# ------------------------------------------------------------------- inputs

def _polydisperse(side, density, seed):
    """A two-kind fluid on a jittered lattice, each particle with its own sigma."""
    n = side * side
    length = math.sqrt(n / density)
    rng = np.random.Generator(np.random.PCG64(seed))
    ij = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="xy"), -1).reshape(-1, 2)
    pos = np.mod((ij + 0.5) * (length / side) + rng.uniform(-0.1, 0.1, size=(n, 2)), length)
    vel = rng.normal(0.0, 1.0, size=(n, 2))
    kind = rng.integers(0, 2, size=n).astype(np.int32)
    sigma = rng.uniform(0.9, 1.05, size=n)
    rc = [2.5, 2.3, 2.3, 2.1]
    sc = S.Scene(meta=dict(N=n, L=length))
    sc.add("init", length, length).add("PBC", 2).add("set_dt", 0.005).add("set_numTypes", 2)
    sc.add("set_pair_potential", [1.0, 0.8, 0.8, 0.6], rc, [S.lj_shift(r) for r in rc])
    sc.add("set_skin", 0.3)
    sc.add("add_particles", pos[:, 0], pos[:, 1], vel[:, 0], vel[:, 1], np.ones(n), sigma, kind)
    sc.add("init_neighbor_list")
    return sc


def _wall_speed_strain(side, steps):
    """The strain of compression() at which its wall moves at 5 sigma / tau."""
    return 5.0 * steps * 0.002 / math.sqrt(side * side * math.pi * 25.0 / 0.5)


def _replica_sizes(case):
    """The ensemble's atom counts: log-uniform, the same for every seed."""
    rng = np.random.Generator(np.random.PCG64(8))
    return np.rint(np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]),
                                      size=case["replicas"]))).astype(int)


def _scenes(case, seed):
    """The scenes of a case: one, or one per replica."""
    if case["kind"] == "forces":
        return [_polydisperse(case["side"], case["density"], 7 * seed + 1)]
    if case["kind"] == "batch":
        rng = np.random.Generator(np.random.PCG64(7 * seed + 2))
        n, sizes = case["replicas"], _replica_sizes(case)
        dens, temps = rng.uniform(0.6, 0.85, size=n), rng.uniform(0.1, 1.5, size=n)
        mesh = S.hex_disk_mesh(5.0, 6, jitter=0.02, seed=3)
        return [S.mixed_replica(int(sizes[r]), float(dens[r]), float(temps[r]), seed=1000 * seed + r, mesh=mesh)
                for r in range(n)]
    if case["kind"] == "adjoint":
        return [S.compression(n_side=case["side"], steps=case["steps"],
                              strain=_wall_speed_strain(case["side"], case["steps"]),
                              seeds=(3, 7 * seed + 1, 7 * seed + 2, 7 * seed + 3))]
    if case["system"] == "lj":
        return [S.lj_fluid(n_side=case["side"], density=case["density"], T=case["T"], seed_pos=7 * seed + 1,
                           seed_vel=7 * seed + 2)]
    if case["system"] == "suspension":
        return [S.suspension(n_side=case["side"], seeds=(3, 7 * seed + 1, 7 * seed + 2))]
    return [S.large_mixed(n_side=case["side"], n_solvent=case["solvent"],
                          seeds=(3, 7 * seed + 1, 7 * seed + 2, 7 * seed + 3))]


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).pin_memory()


def _program(sc, mode):
    """A system set up for its runs, its start state and its result buffers."""
    s = F.System()
    s.set_force_mode(mode)
    sc.replay(s)
    pos, vel, _ = s.get_state()
    s.allocate_cuda()
    out = {k: torch.empty((s.N, 2), dtype=torch.float32, pin_memory=True) for k in ("pos", "vel", "acc")}
    return {"system": s, "pos": _pinned(pos), "vel": _pinned(vel), "out": out}


def prepare(case, seed):
    scenes = _scenes(case, seed)
    progs = [_program(sc, MODES[case.get("mode", "reference")]) for sc in scenes]
    state = {"case": case, "programs": progs}
    if case["kind"] == "batch":
        state["batch"] = F.Batch()
        for p in progs:
            state["batch"].add(p["system"])
    if case["kind"] == "adjoint":
        state["wall"] = next(a for nm, a in scenes[0].calls if nm == "set_moving_wall")
    return state


# -------------------------------------------------------------------- a pass

def _feed(p):
    p["system"].set_state_ptr(p["pos"].data_ptr(), p["vel"].data_ptr())


def _fetch(p):
    o = p["out"]
    p["system"].get_state_ptr(o["pos"].data_ptr(), o["vel"].data_ptr(), o["acc"].data_ptr())
    return o


def _energies(s):
    """U, W and sum m v^2 (sums of single-precision terms), and the rebuilds of the run."""
    e = s.energies()
    return e[:3].astype(np.float32), int(e[5])


def run(state):
    case, progs = state["case"], state["programs"]
    p = progs[0]
    s = p["system"]
    if case["kind"] == "run":
        _feed(p)
        s.run(case["steps"])
        out = dict(_fetch(p))
        out["energies"], out["rebuilds"] = _energies(s)
        return out
    if case["kind"] == "forces":
        _feed(p)
        s.build_nn()
        s.calc_forces()
        return {"forces": s.forces(), "particle_energies": s.particle_energies(),
                "energies": s.energies()[:2].astype(np.float32)}
    if case["kind"] == "batch":
        for q in progs:
            _feed(q)
        state["batch"].run(case["steps"])
        got = [_fetch(q) for q in progs]
        return {k: torch.cat([g[k] for g in got]) for k in ("pos", "vel", "acc")}
    # the wall back at its start, the given state, one forward and backward
    k, y0, v = state["wall"]
    s.set_moving_wall(k, y0 + v * s.steps() * s.get_dt(), v)
    _feed(p)
    s.adjoint_forward(case["steps"], case["every"])
    out = {"observable": np.array(s.adjoint_observable(), np.float32)}
    out.update(s.adjoint_backward(1.0, 1.0))
    return out


# ---------------------------------------------------------------------- work

PAIR_FLOPS, TRI_FLOPS, BOND_FLOPS, ATOM_FLOPS = 27, 140, 20, 20


def work(case):
    """Bytes: per step every atom's position and velocity read and written and
    its mass read, each triangle's and bond's constants; the state handed over
    in host memory at both ends.  Operations: pairs inside the cutoff (each
    once), triangles, bonds, the integration; the backward counts twice the
    forward's terms."""
    disk_atoms, disk_tris, disk_bonds = 127, 216, 36
    if case["kind"] == "batch":
        n = float(_replica_sizes(case).sum())
        disks, solvent, density, steps = 0.1 * n / disk_atoms, 0.9 * n, 0.72, case["steps"]
    elif case["kind"] == "adjoint" or case.get("system") == "suspension":
        disks, solvent, density, steps = case["side"] ** 2, 0, 0.0, case["steps"]
    elif case.get("system") == "mixed":
        disks, solvent, density, steps = case["side"] ** 2, case["solvent"], 0.8, case["steps"]
    else:
        disks, solvent, density, steps = 0, case["side"] ** 2, case["density"], case.get("steps", 1)
    atoms = disks * disk_atoms + solvent
    pairs = solvent * density * math.pi * 2.5 ** 2 / 2
    step_bytes = 36 * atoms + 36 * disks * disk_tris + 12 * disks * disk_bonds
    step_flops = (PAIR_FLOPS * pairs + ATOM_FLOPS * atoms + TRI_FLOPS * disks * disk_tris
                  + BOND_FLOPS * disks * disk_bonds)
    passes = 3 if case["kind"] == "adjoint" else 1
    return {"bytes": 40 * atoms + passes * steps * step_bytes, "flops": passes * steps * step_flops}


# ------------------------------------------- the same results in 64 bits
#
# Plain torch in double precision: pair lists from a cell table (rebuilt when
# the largest displacement could have reached half their skin), the forces by
# index_add, the kick-drift-kick leapfrog.  Inputs are the single-precision
# values that the program hands over.

SKIN64 = 0.5


def _f32(x):
    return float(np.float32(x))


class _Exact:
    """One or more scenes (replicas side by side, each in its own box)."""

    def __init__(self, scenes):
        self.dev = torch.device("cuda")
        d = dict(dtype=torch.float64, device=self.dev)
        parts = [self._read(sc) for sc in scenes]
        a = parts[0]
        self.dt, self.kbond, self.pbc, self.nt = a["dt"], a["kbond"], a["pbc"], a["nt"]
        self.eps, self.rc, self.us = (torch.tensor(a[k], **d) for k in ("eps", "rc", "us"))
        self.first = np.cumsum([0] + [p["pos"].shape[0] for p in parts])
        cat = lambda k: np.concatenate([p[k] for p in parts])  # noqa: E731
        shift = lambda k: np.concatenate([p[k] + f for p, f in zip(parts, self.first)])  # noqa: E731
        self.x0, self.v0 = torch.tensor(cat("pos"), **d), torch.tensor(cat("vel"), **d)
        self.m, self.sig = torch.tensor(cat("mass"), **d), torch.tensor(cat("sigma"), **d)
        self.type = torch.tensor(cat("type"), device=self.dev)
        groups = np.cumsum([0] + [p["disks"] for p in parts])
        self.excl = torch.tensor(np.concatenate([np.where(p["excl"] < 0, -1, p["excl"] + g)
                                                 for p, g in zip(parts, groups)]), device=self.dev)
        self.boxes = [p["L"] for p in parts]
        self.L = torch.tensor(np.concatenate([np.tile(p["L"], (p["pos"].shape[0], 1)) for p in parts]), **d)
        self.bond = torch.tensor(shift("bond"), device=self.dev)
        self.tri = torch.tensor(shift("tri"), device=self.dev)
        self.disk_of_tri = torch.tensor(np.concatenate([p["disk_of_tri"] + g for p, g in zip(parts, groups)]),
                                        device=self.dev)
        ref = torch.tensor(cat("ref"), **d)
        if len(self.bond):
            self.r0 = self._vec(self.x0, self.bond[:, 0], self.bond[:, 1]).norm(dim=1)
        if len(self.tri):
            e1, e2 = ref[self.tri[:, 0]] - ref[self.tri[:, 2]], ref[self.tri[:, 1]] - ref[self.tri[:, 2]]
            det = e1[:, 0] * e2[:, 1] - e2[:, 0] * e1[:, 1]
            self.vol = det / 2
            # inverse of the edge matrix with columns e1, e2
            self.B = (e2[:, 1] / det, -e2[:, 0] / det, -e1[:, 1] / det, e1[:, 0] / det)  # B00 B01 B10 B11
        self.E = torch.tensor(cat("E"), **d)
        self.nu = torch.tensor(cat("nu"), **d)
        self.wall = a["wall"]
        self.log_eps = self.log_sigma = torch.zeros((), **d)

    @staticmethod
    def _read(sc):
        """The arrays that a scene's calls set up."""
        p = dict(kbond=0.0, wall=None, nt=1)
        E = nu = 0.0
        pos, vel, mass, sigma, typ, excl, ref = [], [], [], [], [], [], []
        bond, tri, own, n, disks = [], [], {}, 0, 0
        edges = None
        for nm, a in sc.calls:
            if nm == "init":
                p["L"] = np.array([_f32(a[0]), _f32(a[1])])
            elif nm == "PBC":
                p["pbc"] = a[0]
            elif nm == "set_dt":
                p["dt"] = _f32(a[0])
            elif nm == "set_numTypes":
                p["nt"] = a[0]
            elif nm == "set_pair_potential":
                p["eps"], p["rc"], p["us"] = (np.asarray(v, np.float32).astype(np.float64) for v in a)
            elif nm == "set_kBond":
                p["kbond"] = _f32(a[0])
            elif nm == "set_youngs_modulus":
                E = _f32(a[0])
            elif nm == "set_poisson_ratio":
                nu = _f32(a[0])
            elif nm == "set_elastomer_material":
                own[a[0]] = (_f32(a[1]), _f32(a[2]))
            elif nm == "set_moving_wall":
                p["wall"] = tuple(_f32(v) for v in a)
            elif nm == "add_elastomer":
                verts, t1 = np.asarray(a[0], np.float32), np.asarray(a[1]).reshape(-1, 3) - 1
                x = (verts + np.array([a[2], a[3]], np.float32)).astype(np.float64)
                if edges is None:
                    every = np.sort(np.concatenate([t1[:, [0, 1]], t1[:, [0, 2]], t1[:, [1, 2]]]), axis=1)
                    uniq, cnt = np.unique(every, axis=0, return_counts=True)
                    edges = uniq[cnt == 1]
                area = lambda y: 0.5 * ((y[t1[:, 2], 1] - y[t1[:, 0], 1]) * (y[t1[:, 1], 0] - y[t1[:, 0], 0])  # noqa: E731
                                        - (y[t1[:, 1], 1] - y[t1[:, 0], 1]) * (y[t1[:, 2], 0] - y[t1[:, 0], 0]))
                vol = area(x)
                if disks == 0:
                    first = vol  # the masses use the first disk's areas (femmd2D/src/particles.cpp:364)
                m = np.zeros(len(x))
                np.add.at(m, t1.ravel(), np.repeat(_f32(a[7]) / vol.sum() * first / 3, 3))
                pos.append(x)
                ref.append(x)
                mass.append(m)
                sigma.append(np.full(len(x), _f32(a[6])))
                typ.append(np.full(len(x), a[4]))
                excl.append(np.full(len(x), disks))
                bond.append(edges + n)
                tri.append(t1 + n)
                n += len(x)
                disks += 1
            elif nm == "add_particles":
                q = np.stack([np.asarray(a[0], np.float32), np.asarray(a[1], np.float32)], 1).astype(np.float64)
                pos.append(q)
                ref.append(np.zeros_like(q))
                vel = [np.zeros((n, 2)), np.stack([np.asarray(a[2], np.float32), np.asarray(a[3], np.float32)],
                                                  1).astype(np.float64)]
                mass.append(np.asarray(a[4], np.float32).astype(np.float64))
                sigma.append(np.asarray(a[5], np.float32).astype(np.float64))
                typ.append(np.asarray(a[6]))
                excl.append(np.full(len(q), -1))
                n += len(q)
            elif nm == "set_velocities_array":
                vel = [np.asarray(a[0], np.float32).astype(np.float64)]
        none2, none3 = np.zeros((0, 2), np.int64), np.zeros((0, 3), np.int64)
        p.update(pos=np.concatenate(pos), vel=np.concatenate(vel), mass=np.concatenate(mass), ref=np.concatenate(ref),
                 sigma=np.concatenate(sigma), type=np.concatenate(typ).astype(np.int64),
                 excl=np.concatenate(excl).astype(np.int64), bond=np.concatenate(bond) if disks else none2,
                 tri=np.concatenate(tri) if disks else none3, disks=disks,
                 disk_of_tri=np.repeat(np.arange(disks), len(tri[0]) if disks else 0),
                 E=np.array([own.get(e, (E, nu))[0] for e in range(disks)]),
                 nu=np.array([own.get(e, (E, nu))[1] for e in range(disks)]))
        return p

    # differences across the periodic axes
    def _vec(self, x, i, j, every_axis=False):
        d = x[i] - x[j]
        k = torch.round(d.detach() / self.L[i])
        if not every_axis and self.pbc < 2:
            k = k * torch.tensor([1.0 if self.pbc == 1 else 0.0, 0.0], dtype=k.dtype, device=k.device)
        return d - k * self.L[i]

    def _wrap(self, x):
        w = x - torch.floor(x.detach() / self.L) * self.L
        if self.pbc == 2:
            return w
        return torch.stack([w[:, 0], x[:, 1]], 1) if self.pbc == 1 else x

    def _pairs(self, x):
        """Pairs i < j within the largest cutoff + the skin, not of one disk."""
        reach = float((self.rc.max() * self.sig.max()).item()) + SKIN64
        found = []
        for b, L in enumerate(self.boxes):
            lo, hi = int(self.first[b]), int(self.first[b + 1])
            y, n = x[lo:hi], hi - lo
            nc = [max(int(L[q] / reach), 1) for q in (0, 1)]
            if min(nc) < 3:
                i, j = torch.triu_indices(n, n, 1, device=self.dev)
                found.append(self._near(x, i + lo, j + lo, reach))
                continue
            c = [torch.clamp((y[:, q] / L[q] * nc[q]).long(), 0, nc[q] - 1) for q in (0, 1)]
            cell = c[0] * nc[1] + c[1]
            order = torch.argsort(cell)
            count = torch.bincount(cell, minlength=nc[0] * nc[1])
            start = torch.cumsum(count, 0) - count
            cap = int(count.max().item())
            table = torch.full((nc[0] * nc[1], cap), n, device=self.dev)
            slot = torch.arange(n, device=self.dev) - start[cell[order]]
            table[cell[order], slot] = order
            for p in range(0, n, 200000):
                me = torch.arange(p, min(p + 200000, n), device=self.dev)
                for dx in (-1, 0, 1):
                    for dy in (-1, 0, 1):
                        near = ((c[0][me] + dx) % nc[0]) * nc[1] + (c[1][me] + dy) % nc[1]
                        cand = table[near]
                        r, q = torch.nonzero((cand < n) & (cand > me[:, None]), as_tuple=True)
                        found.append(self._near(x, me[r] + lo, cand[r, q] + lo, reach))
        return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])

    def _near(self, x, i, j, reach):
        keep = (self._vec(x, i, j) ** 2).sum(1) <= reach * reach
        keep &= (self.excl[i] < 0) | (self.excl[i] != self.excl[j])
        return i[keep], j[keep]

    def forces(self, x, pairs, n=0, energy=False):
        """Forces (and, with energy, the energy per particle, the sum W of f.r and the triangle energy)."""
        f = torch.zeros_like(x)
        u = torch.zeros_like(x[:, 0])
        W = 0.0
        scale = torch.exp(self.log_sigma)
        i, j = pairs
        d = self._vec(x, i, j)
        t = self.type[i] * self.nt + self.type[j]
        s2 = ((self.sig[i] + self.sig[j]) / 2 * scale) ** 2
        r2 = (d * d).sum(1)
        inside = torch.nonzero(r2.detach() < self.rc[t] ** 2 * s2.detach()).squeeze(1)
        i, j, d, t, s2, r2 = i[inside], j[inside], d[inside], t[inside], s2[inside], r2[inside]
        eps = self.eps[t] * torch.exp(self.log_eps)
        q2 = s2 / r2
        q6 = q2 ** 3
        fc = 48 * eps / s2 * q6 * (q6 - 0.5) * q2
        g = fc[:, None] * d
        f = f.index_add(0, i, g).index_add(0, j, -g)
        if energy:
            up = 4 * eps * q6 * (q6 - 1) + self.us[t]
            u = u.index_add(0, i, up / 2).index_add(0, j, up / 2)
            W = (fc * r2).sum()
        if len(self.bond) and self.kbond > 0:
            i, j = self.bond[:, 0], self.bond[:, 1]
            d = self._vec(x, i, j)
            r = d.norm(dim=1)
            g = (-self.kbond * (r - self.r0) / r)[:, None] * d
            f = f.index_add(0, i, g).index_add(0, j, -g)
            if energy:
                u = u.index_add(0, i, 0.5 * self.kbond * (r - self.r0) ** 2)
        fea = 0.0
        if len(self.tri):
            a, b, c = self.tri.unbind(1)
            p, q = self._vec(x, a, c, True), self._vec(x, b, c, True)
            B00, B01, B10, B11 = self.B
            F00, F10 = p[:, 0] * B00 + q[:, 0] * B10, p[:, 1] * B00 + q[:, 1] * B10
            F01, F11 = p[:, 0] * B01 + q[:, 0] * B11, p[:, 1] * B01 + q[:, 1] * B11
            J = F00 * F11 - F01 * F10
            E, nu = self.E[self.disk_of_tri], self.nu[self.disk_of_tri]
            mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
            lj = torch.log(J)
            k = lam * lj - mu
            # P = mu F + (lam ln J - mu) F^-T, nodal forces -vol P B^T
            P00, P10 = mu * F00 + k * F11 / J, mu * F10 - k * F01 / J
            P01, P11 = mu * F01 - k * F10 / J, mu * F11 + k * F00 / J
            h0 = -self.vol[:, None] * torch.stack([P00 * B00 + P01 * B01, P10 * B00 + P11 * B01], 1)
            h1 = -self.vol[:, None] * torch.stack([P00 * B10 + P01 * B11, P10 * B10 + P11 * B11], 1)
            f = f.index_add(0, a, h0).index_add(0, b, h1).index_add(0, c, -h0 - h1)
            if energy:
                i1 = F00 ** 2 + F01 ** 2 + F10 ** 2 + F11 ** 2
                e = self.vol * (0.5 * mu * (i1 - 2 - 2 * lj) + 0.5 * lam * lj ** 2)
                fea = e.sum()
                for v in (a, b, c):
                    u = u.index_add(0, v, e / 3)
        if self.wall is not None:
            k, top, bottom = self._walls(x, n)
            f = f + torch.stack([torch.zeros_like(top), k * (bottom - top)], 1)
            if energy:
                u = u + 0.5 * k * (top ** 2 + bottom ** 2)
        return (f, u, W, fea) if energy else f

    def _walls(self, x, n):
        """The walls' stiffness and every particle's overlap with the top and the bottom one."""
        k, y0, v = self.wall
        reach = 2.0 ** (1.0 / 6.0) * self.sig * torch.exp(self.log_sigma)
        yw = y0 - v * (n * self.dt)
        return k, torch.relu(x[:, 1] + reach - yw), torch.relu(reach - x[:, 1])

    def trajectory(self, steps):
        """x, v, a after run(steps), and the pairs in reach of x."""
        x, v = self._wrap(self.x0) if self.pbc == 2 else self.x0, self.v0
        pairs, moved = self._pairs(x.detach()), 0.0
        a = self.forces(x, pairs, 0) / self.m[:, None]
        for n in range(1, steps + 1):
            v = v + 0.5 * self.dt * a
            x = self._wrap(x + self.dt * v)
            moved += self.dt * float(v.detach().norm(dim=1).max().item())
            if 2.0 * moved > 0.95 * SKIN64:
                pairs, moved = self._pairs(x.detach()), 0.0
            a = self.forces(x, pairs, n) / self.m[:, None]
            v = v + 0.5 * self.dt * a
        return x, v, a, pairs


def exact(case, seed):
    ex = _Exact(_scenes(case, seed))
    if case["kind"] == "forces":
        f, u, W, _ = ex.forces(ex.x0, ex._pairs(ex.x0), energy=True)
        return {"forces": f, "particle_energies": u, "energies": torch.stack([u.sum(), W])}
    if case["kind"] == "adjoint":
        leaves = {"x0": ex.x0, "v0": ex.v0, "E": ex.E, "nu": ex.nu, "log_eps": ex.log_eps.clone(),
                  "log_sigma": ex.log_sigma.clone()}
        for t in leaves.values():
            t.requires_grad_(True)
        ex.log_eps, ex.log_sigma = leaves["log_eps"], leaves["log_sigma"]
        x, _, _, pairs = ex.trajectory(case["steps"])
        fea = ex.forces(x, pairs, case["steps"], energy=True)[3]
        k, top, bottom = ex._walls(x, case["steps"])
        stress = k * (top.sum() + bottom.sum()) / (2 * ex.boxes[0][0])
        grads = torch.autograd.grad(stress + fea, list(leaves.values()))
        out = {name: g.detach() for name, g in zip(leaves, grads)}
        out["observable"] = torch.stack([stress, fea]).detach()
        out["log_eps"], out["log_sigma"] = float(out["log_eps"]), float(out["log_sigma"])
        return out
    x, v, a, pairs = ex.trajectory(case["steps"])
    out = {"pos": x, "vel": v, "acc": a}
    if case["kind"] == "run":
        _, u, W, _ = ex.forces(x, pairs, case["steps"], energy=True)
        out["energies"] = torch.stack([u.sum(), W, (ex.m * (v * v).sum(1)).sum()])
        out["rebuilds"] = None
    return out
