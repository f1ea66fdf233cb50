"""Triangles by block in the whole-run launch (k_coop.cuh): every block works
all the triangles of its own particles.  Against the same run through the plain
kernels (direct launches), bit for bit, as in test_gpu_coop.py.

Cases: one tile of particles a block, two neighbouring tiles a block (more than
one tile per SM: 168 and 304 tiles on 152 SMs), more than two, disks in
solvent on two tiles a block, a vertex of more triangles than a block keeps at
hand (16 > 8: the triangle pass apart), the Green strain law, and the triangle
forces turned off and on between runs.
"""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S

pytestmark = pytest.mark.gpu


def fan(spokes, radius=5.0):
    """A disk of one inner vertex with 'spokes' triangles around it."""
    t = 2 * np.pi * np.arange(spokes) / spokes
    pts = np.concatenate([[[0.0, 0.0]], radius * np.stack([np.cos(t), np.sin(t)], -1)])
    k = np.arange(spokes)
    return pts, np.stack([np.zeros(spokes, int), 1 + k, 1 + (k + 1) % spokes], -1) + 1


CASES = {
    "one_tile": (lambda: S.suspension(n_side=5, T=0.5), 0),
    "pairs": (lambda: S.suspension(n_side=13, T=0.5), 0),
    "pairs_full": (lambda: S.suspension(n_side=17, T=0.5), 0),
    "three_tiles": (lambda: S.suspension(n_side=20, T=0.5), 0),
    "mixed_pairs": (lambda: S.large_mixed(n_side=6, n_solvent=25000), 0),
    "fan": (lambda: S.mixed_replica(3000, 0.7, 0.5, seed=4, mesh=fan(16)), 0),
    "green": (lambda: S.suspension(n_side=13, T=0.5), 1),
}


def record(make, direct, law):
    s = F.System()
    s.set_fea_law(law)
    make().replay(s)
    s.set_profiling(direct)
    out = []
    for n, E in ((1, 50.0), (2, 50.0), (3, 0.0), (33, 50.0)):
        s.set_youngs_modulus(E)
        s.run(n)
        out += [*s.get_state(), s.forces(), s.energies(), s.step_observables()]
    s.set_profiling(False)
    return out


@pytest.mark.parametrize("name", CASES)
def test_triangles_by_block_equal_plain_kernels(name):
    make, law = CASES[name]
    for a, b in zip(record(make, False, law), record(make, True, law)):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))
