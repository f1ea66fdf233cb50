"""Gases in large boxes, far more cells than particles: the fast mode's small
fluids run in one launch up to the cells whose starts a block holds (39,264); beyond
that and in the reference mode the plain kernels take a box of more than 4096
cells and four a particle.  Against the plain kernels (direct launches) bit for
bit, the per-step energies among it but for the fast launch beyond 39,264 cells,
which groups them by id; with and without trajectory frames."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from test_gpu_coop import ragged_fluid

pytestmark = pytest.mark.gpu

# particles, cells along an edge of the box (of 2.8 and a little more)
CASES = [(1, 3), (64, 90), (129, 68), (2000, 159), (16384, 198), (16384, 199), (700, 250)]
BY_ID = (16384, 199)


def record(n, cells, mode, direct, path):
    s = F.System()
    s.set_force_mode(mode)
    side = int(np.ceil(np.sqrt(n)))
    ragged_fluid(n, density=(side / (2.8001 * cells)) ** 2).replay(s)
    if path:
        s.set_trajectory(path, 6)
    s.set_profiling(direct)
    out = []
    for steps in (1, 40, 9):
        s.run(steps)
        out += [*s.get_state(), s.forces(), s.step_observables(), np.array([s.total_updates()])]
        start, ids = s.cells()
        assert len(start) == cells * cells + 1
        out += [start, ids]
    s.set_profiling(False)
    if path:
        s.flush_trajectory()
        out.append(np.frombuffer(path.read_bytes(), np.uint8))
    return out


@pytest.mark.parametrize("frames", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,cells", CASES)
def test_dilute_runs_equal_plain_kernels(n, cells, mode, frames, tmp_path):
    a, b = (record(n, cells, mode, direct, tmp_path / f"{direct}.vtf" if frames else None) for direct in (False, True))
    for x, y in zip(a, b):
        if mode == 1 and (n, cells) == BY_ID and x.ndim == 2 and x.shape[1] == 6:
            x, y = x[:, 3:], y[:, 3:]
        x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
        assert x.shape == y.shape and np.array_equal(x.view(np.uint8), y.view(np.uint8))
