"""Whole-run launches of the fast mode's small systems and of runs with
trajectory frames (one launch from a frame to the next) against the plain kernels
(direct launches): the frames' bytes, the state, the rebuilds and the per-step
observables.  The same operations and the same 128-slot energy groups, so all
bit for bit, but for the energies of fast-mode systems above 128 tiles of 128
particles or with bonded particles, which are grouped by id there (checked
elsewhere).

Sizes: a tile, one particle more, the largest system grouped by slot (16,384)
and one beyond it; frames at every step, at and next to rebuilds, at the end.
"""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S
from test_gpu_coop import ragged_fluid, resized

pytestmark = pytest.mark.gpu

CASES = {
    "tile": (lambda: ragged_fluid(128), "fast", 5, (1, 4, 40)),
    "tile_and_one": (lambda: ragged_fluid(129), "fast", 1, (3, 12)),
    "sigma": (lambda: resized(ragged_fluid(2100, density=0.75), 1.1), "fast", 9, (36, 18)),
    "largest_by_slot": (lambda: ragged_fluid(16384), "fast", 15, (30, 7)),
    "beyond": (lambda: ragged_fluid(16385), "fast", 15, (30, 7)),
    "mixed": (lambda: S.large_mixed(n_side=5, n_solvent=7001), "fast", 10, (35,)),
    "reference": (lambda: ragged_fluid(5000), "reference", 7, (1, 40, 8)),
    "disks": (lambda: S.suspension(n_side=9, T=0.5), "reference", 4, (17,)),
    "no_frames": (lambda: ragged_fluid(700), "fast", 0, (1, 2, 60)),
}
MODES = {"reference": 0, "fast": 1}


def record(make, mode, every, runs, direct, path):
    s = F.System()
    s.set_force_mode(MODES[mode])
    make().replay(s)
    s.run(0)
    if every:
        s.set_trajectory(path, every)
    s.set_profiling(direct)
    out = []
    for n in runs:
        s.run(n)
        out += [*s.get_state(), s.forces(), np.array([s.total_updates(), s.steps()]), s.step_observables()]
    s.set_profiling(False)
    if every:
        s.flush_trajectory()
        out.append(np.frombuffer(path.read_bytes(), np.uint8))
    return out


@pytest.mark.parametrize("name", CASES)
def test_launches_from_frame_to_frame_equal_plain_kernels(name, tmp_path):
    make, mode, every, runs = CASES[name]
    a = record(make, mode, every, runs, False, tmp_path / "a.vtf")
    b = record(make, mode, every, runs, True, tmp_path / "b.vtf")
    by_id = name in ("beyond", "mixed")
    for x, y in zip(a, b):
        if by_id and x.ndim == 2 and x.shape[1] == 6:
            x, y = x[:, 3:], y[:, 3:]
        x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
        assert x.shape == y.shape and np.array_equal(x.view(np.uint8), y.view(np.uint8))
