"""A run in one cooperative launch (k_coop.cu) against the same run through
the plain step and rebuild kernels (direct launches, set_profiling), bit for
bit: positions, velocities, accelerations, forces, the energies, the per-step
observables, the rebuild count, cells and neighbour lists.  Both paths do the
same single-precision operations in the same order and add the same 128- and
256-wide partial sums in fixed point, so no tolerance applies.

Sizes: below, at and above one block (1024 particles), a tile edge (128)
and one particle beyond it, a grid of fewer than five cells (the general
list walk), elastomers (triangle pass), two types with a size per particle,
fixed walls, and moving walls (the step index inside the launch).
"""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S

pytestmark = pytest.mark.gpu


def ragged_fluid(n, density=0.75, pbc=2, types=1, own_sigma=False, seed=5):
    """n particles on a jittered lattice (any n), optionally of two types."""
    rng = np.random.Generator(np.random.PCG64(seed))
    side = int(np.ceil(np.sqrt(n)))
    a = float(1.0 / np.sqrt(density))
    # walls start outside the particles' repulsion: room of one sigma where the box is not periodic
    room = 0.0 if pbc == 2 else 1.0
    length = side * a + 2 * room
    ij = np.stack(np.meshgrid(np.arange(side), np.arange(side)), -1).reshape(-1, 2)[:n]
    x = room + (ij + 0.5) * a + rng.uniform(-0.1, 0.1, (n, 2))
    v = rng.normal(0.0, 1.0, (n, 2))
    t = rng.integers(0, types, n).astype(np.int32)
    sig = rng.uniform(0.9, 1.05, n) if own_sigma else np.ones(n)
    sc = S.Scene(meta=dict(N=n))
    sc.add("init", length, length).add("PBC", pbc).add("set_dt", 0.005).add("set_numTypes", types)
    rc = [2.5] if types == 1 else [2.5, 2.3, 2.3, 2.1]
    sc.add("set_pair_potential", [1.0] * len(rc), rc, [S.lj_shift(r) for r in rc]).add("set_skin", 0.3)
    sc.add("add_particles", x[:, 0], x[:, 1], v[:, 0], v[:, 1], np.ones(n), sig, t).add("init_neighbor_list")
    return sc


SCENES = {
    "four_cells": lambda: ragged_fluid(100),
    "tile": lambda: ragged_fluid(128),
    "tile_and_one": lambda: ragged_fluid(1025),
    "one_block": lambda: ragged_fluid(1024),
    "many_tiles": lambda: ragged_fluid(30001),
    "two_types_sigma": lambda: ragged_fluid(5003, density=0.65, types=2, own_sigma=True),
    "two_types": lambda: ragged_fluid(2300, types=2),
    "x_periodic": lambda: ragged_fluid(1500, density=0.6, pbc=1),
    "walls": lambda: ragged_fluid(1500, density=0.6, pbc=0),
    "disks_one_block": lambda: S.suspension(n_side=2),
    "disks": lambda: S.suspension(n_side=9, T=0.5),
    "mixed": lambda: S.large_mixed(n_side=5, n_solvent=7001),
    "moving_wall": lambda: S.compression(n_side=4),
}


def record(sc, direct, runs):
    s = F.System()
    sc.replay(s)
    s.set_profiling(direct)
    out = []
    for n in runs:
        s.run(n)
        out += [*s.get_state(), s.forces(), s.energies(), s.step_observables(), *s.cells(), *s.neighbors()]
    s.set_profiling(False)
    return out


@pytest.mark.parametrize("name", SCENES)
def test_one_launch_equals_plain_kernels(name):
    sc = SCENES[name]()
    runs = (1, 2, 33, 20)
    for a, b in zip(record(sc, False, runs), record(sc, True, runs)):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


def rows_as_sets(start, lst):
    rows = np.repeat(np.arange(len(start) - 1), np.diff(start))
    return lst[np.lexsort((lst, rows))]


FAST_SCENES = {
    "one_type": lambda: ragged_fluid(16385),
    "one_type_sigma": lambda: resized(ragged_fluid(17003, density=0.75), 1.1),
    "x_periodic": lambda: ragged_fluid(1500, density=0.6, pbc=1),
    "walls": lambda: ragged_fluid(700, density=0.6, pbc=0),
    "two_types": lambda: ragged_fluid(2300, types=2),
    "disks": lambda: S.suspension(n_side=9, T=0.5),
    "mixed": lambda: S.large_mixed(n_side=5, n_solvent=7001),
}


def resized(sc, sigma):
    """Every sigma and length of a scene's fluid scaled by 'sigma'."""
    def call(name, a):
        if name == "init":
            return name, (a[0] * sigma, a[1] * sigma)
        if name == "add_particles":
            return name, (a[0] * sigma, a[1] * sigma, *a[2:5], a[5] * sigma, a[6])
        return name, a
    sc.calls = [call(n, a) for n, a in sc.calls]
    return sc


@pytest.mark.parametrize("name", FAST_SCENES)
def test_fast_mode_one_launch_equals_its_kernels(name):
    """The fast mode's whole-run launch against its step and rebuild kernels:
    state, forces, largest speeds, rebuilds and cells bit for bit, neighbour
    sets equal.  The energies are sums of the same single-precision terms in
    other groups: each group adds at most 128 terms one by one or 64 sums of
    such groups, so a total is within 192 * 2^-24 = 1.2e-5 of the sum of its
    terms' magnitudes, for which the particles' own |energy| bound stands in."""
    sc = FAST_SCENES[name]()
    systems = []
    for direct in (False, True):
        s = F.System()
        s.set_force_mode(1)
        sc.replay(s)
        s.set_profiling(direct)
        systems.append(s)
    for n in (1, 2, 33, 20):
        got = []
        for s in systems:
            s.run(n)
            st, lst = s.neighbors()
            got.append(dict(exact=[*s.get_state(), s.forces(), s.step_observables()[:, 3:], *s.cells(), st,
                                   rows_as_sets(st, lst)], obs=s.step_observables(), updates=s.total_updates()))
        for a, b in zip(got[0]["exact"], got[1]["exact"]):
            assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))
        assert got[0]["updates"] == got[1]["updates"]
        for s in systems:
            s.calc_forces()  # over the lists that the run left behind
        fa, fb = (s.forces() for s in systems)
        assert np.array_equal(fa.view(np.uint32), fb.view(np.uint32))
        scale = max(np.abs(systems[0].particle_energies()).sum(), np.abs(got[0]["obs"][:, :3]).max())
        assert np.abs(got[0]["obs"][:, :3] - got[1]["obs"][:, :3]).max() <= 1.2e-5 * scale


def test_list_overflow_repeats_the_run():
    """Lists outgrown inside the launch: the run is rolled back and repeated."""
    sc = ragged_fluid(3000)
    a, b = F.System(), F.System()
    for s in (a, b):
        sc.replay(s)
    a.allocate_cuda()
    a.set_neighbor_capacity(4)
    for s in (a, b):
        s.run(30)
    assert a.neighbor_capacity() > 4
    for x, y in zip(a.get_state(), b.get_state()):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


def test_expired_exchange_reports_and_recovers():
    """A grid-wide exchange that gives up (bounded wait) ends the run with
    FEMMD_TIMEOUT; the context then runs like a fresh one."""
    sc = ragged_fluid(4001)
    s, ref = F.System(), F.System()
    for q in (s, ref):
        sc.replay(q)
    pos, vel, _ = s.get_state()
    s.allocate_cuda()
    s.test_expire_next_exchange()
    with pytest.raises(F.FemmdError) as e:
        s.run(10)
    assert "expired" in str(e.value)
    s.set_state(pos, vel)
    s.run(10)
    ref.run(10)
    for x, y in zip(s.get_state(), ref.get_state()):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
