"""Runs in one cooperative launch (k_coop.cuh) that meet a state the launch cannot
list: a cell of more than 32 particles or a non-finite position.  The launch is left at
that rebuild and the run repeated by the plain kernels, so everything equals
the plain kernels' (direct launches) bit for bit.

Cases: cells crowded from the start (particles much smaller than the list
radius, which does not scale with sigma), crowded only at a later rebuild (an
inward flow), the same with trajectory frames before and after it; NaN and
infinite positions in the start state (the error, again on a second run, and the
context usable afterwards), and NaN velocities (met inside the run).
"""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S
from test_gpu_coop import ragged_fluid

pytestmark = pytest.mark.gpu
MODES = {"reference": 0, "fast": 1}
CELL_CAP = 32


def small_particles(side, a, sigma, inward, dt, seed=3):
    """side^2 particles of the given sigma on a lattice of constant a, with
    thermal velocities, or flowing towards the centre."""
    rng = np.random.Generator(np.random.PCG64(seed))
    ij = np.stack(np.meshgrid(np.arange(side), np.arange(side)), -1).reshape(-1, 2)
    x = (ij + 0.5) * a + rng.uniform(-0.02, 0.02, ij.shape)
    v = rng.normal(0.0, 0.5, ij.shape) - inward * (x - 0.5 * side * a)
    n = len(x)
    sc = S.Scene(meta=dict(N=n))
    sc.add("init", side * a, side * a).add("PBC", 2).add("set_dt", dt).add("set_numTypes", 1)
    sc.add("set_pair_potential", [1.0], [2.5], [S.lj_shift(2.5)]).add("set_skin", 0.3)
    sc.add("add_particles", x[:, 0], x[:, 1], v[:, 0], v[:, 1], np.ones(n), np.full(n, sigma), np.zeros(n, np.int32))
    return sc.add("init_neighbor_list"), side * a


def most_per_cell(pos, box, radius=2.8):
    n = int(box // radius)
    c = np.minimum((pos * n / box).astype(int), n - 1)
    return np.bincount(c[:, 0] * n + c[:, 1]).max()


def record(sc, mode, direct, runs, path=None, every=0, builds=False):
    s = F.System()
    s.set_force_mode(MODES[mode])
    sc.replay(s)
    if path:
        s.set_trajectory(path, every)
    s.set_profiling(direct)
    out = []
    for n in runs:
        s.run(n)
        out += [*s.get_state(), s.forces(), s.step_observables(), *s.cells(), *s.neighbors(),
                np.array([s.total_updates(), s.steps()])]
    s.set_profiling(False)
    if builds:  # (a run repeated with longer lists counts its builds twice: not where the lists grow)
        out.append(np.array([s.nn_stats()["builds"]]))
    if path:
        s.flush_trajectory()
        out.append(np.frombuffer(path.read_bytes(), np.uint8))
    return out


def same_bytes(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
        assert x.shape == y.shape and np.array_equal(x.view(np.uint8), y.view(np.uint8))


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("side", [45, 140])
def test_cells_crowded_from_the_start(mode, side):
    # sigma 0.4 at rho sigma^2 = 0.8: 39 particles per cell of the list radius
    sc, box = small_particles(side, 0.4472, 0.4, 0.0, 0.002)
    runs = (1, 2, 25)
    a, b = (record(sc, mode, direct, runs, builds=True) for direct in (False, True))
    assert most_per_cell(a[0], box) > CELL_CAP
    same_bytes(a, b)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("frames", [False, True])
def test_cells_crowded_later(mode, frames, tmp_path):
    # 25 particles per cell at the start, gathering at the centre of the box
    sc, box = small_particles(40, 0.565, 0.3, 1.2, 0.001)
    start = F.System()
    sc.replay(start)
    assert most_per_cell(start.get_state()[0], box) <= CELL_CAP
    a, b = (record(sc, mode, direct, (300, 5), tmp_path / f"{direct}.vtf" if frames else None, 20)
            for direct in (False, True))
    assert most_per_cell(a[0], box) > CELL_CAP
    same_bytes(a, b)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("first", [0, 7])
def test_non_finite_start_state(mode, value, first):
    """first: steps run before the state is set (0: no list has been built yet)."""
    sc = ragged_fluid(4001)
    s, ref = F.System(), F.System()
    for q in (s, ref):
        q.set_force_mode(MODES[mode])
        sc.replay(q)
    pos, vel, _ = s.get_state()
    s.allocate_cuda()
    if first:
        s.run(first)
    bad = pos.copy()
    bad[1234, 1] = value
    s.set_state(bad, vel)
    for _ in range(2):
        with pytest.raises(F.FemmdError) as e:
            s.run(10)
        assert "NaN or infinite" in str(e.value)
    s.set_state(pos, vel)
    s.run(10)
    ref.run(10)
    for x, y in zip(s.get_state(), ref.get_state()):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


def test_non_finite_inside_the_run():
    """Velocities that become non-finite positions after the first step: the state
    left behind is the plain kernels'."""
    sc = ragged_fluid(2300)
    left = []
    for direct in (False, True):
        s = F.System()
        sc.replay(s)
        pos, vel, _ = s.get_state()
        s.allocate_cuda()
        s.run(3)
        vel[77] = np.nan
        s.set_state(pos, vel)
        s.set_profiling(direct)
        with pytest.raises(F.FemmdError):
            s.run(60)
        left.append([np.isnan(x) for x in s.get_state()] + [np.nan_to_num(x) for x in s.get_state()] +
                    [np.array([s.nn_stats()["builds"]])])
        s.set_profiling(False)
    same_bytes(*left)
