"""Positions at the edge of the box in the whole-run launch against the plain
kernels, bit for bit: -0, and negative coordinates so small that r / L rounds to
-0, which the reference's r - floor(r / L) L leaves where they are.  The
particles of interest have no neighbours."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S

pytestmark = pytest.mark.gpu
L = 50.0
DT = 0.005
TINY = float(np.float32(1.4e-45))  # the smallest float

# x and the displacement of the first drift
CASES = [(-0.0, 0.0), (-0.0, -0.0), (0.0, -0.0), (0.0, -7 * TINY), (0.0, 7 * TINY), (0.0, -30 * TINY),
         (0.0, -1e-40), (0.0, -1e-38), (0.0, -1e-30), (0.0, -1e-29), (0.0, -1e-20), (0.0, -1e-6),
         (float(np.nextafter(np.float32(L), np.float32(0))), 1e-5), (L, 0.0), (L, -1e-20)]


@pytest.mark.parametrize("axis", [0, 1])
def test_edges_of_the_box(axis):
    n = len(CASES)
    x = np.full((n, 2), 25.0)
    x[:, 1 - axis] = 1.5 + 3.1 * np.arange(n)  # apart by more than the cutoff
    v = np.zeros((n, 2))
    sc = S.Scene(meta=dict(N=n))
    sc.add("init", L, L).add("PBC", 2).add("set_dt", DT).add("set_numTypes", 1)
    sc.add("set_pair_potential", [1.0], [2.5], [S.lj_shift(2.5)]).add("set_skin", 0.3)
    sc.add("add_particles", x[:, 0], x[:, 1], v[:, 0], v[:, 1], np.ones(n), np.ones(n), np.zeros(n, np.int32))
    sc.add("init_neighbor_list")
    pos, vel = x.astype(np.float32), v.astype(np.float32)
    with np.errstate(under="ignore"):
        pos[:, axis] = [p for p, _ in CASES]
        vel[:, axis] = [np.float32(d / DT) for _, d in CASES]
    out = []
    for direct in (False, True):
        s = F.System()
        sc.replay(s)
        s.allocate_cuda()
        s.set_state(pos, vel)
        s.set_profiling(direct)
        out.append([])
        for n in (1, 2, 5):
            s.run(n)
            out[-1] += [a.view(np.uint32) for a in s.get_state()]
        s.set_profiling(False)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
