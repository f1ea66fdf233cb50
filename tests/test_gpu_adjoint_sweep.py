"""The reverse steps in one cooperative launch per list (k_adj_sweep) against
two kernels a step (set_profiling): both do the same operations in the same
order, so the gradients, the parameter derivatives and the state left behind are
equal bit for bit.

Cases: one block and one particle beyond it, lists of several rounds (12
entries) with one and two types and a size per particle, walls, elastomers on
one, two neighbouring and three tiles a block, a vertex of more triangles than
the launch keeps at hand (the two kernels), segments of one step, and segments
with several lists.
"""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S
from test_gpu_coop import ragged_fluid
from test_gpu_coop_tri import fan

pytestmark = pytest.mark.gpu

CASES = {
    "one_block": (lambda: ragged_fluid(128), 12, 5),
    "block_and_one": (lambda: ragged_fluid(129), 7, 7),
    "fluid_many_lists": (lambda: ragged_fluid(5000), 70, 35),
    "fluid_three_tiles": (lambda: ragged_fluid(40001), 4, 4),
    "two_types_sigma": (lambda: ragged_fluid(5003, density=0.65, types=2, own_sigma=True), 30, 15),
    "two_types": (lambda: ragged_fluid(2300, types=2), 6, 1),
    "moving_wall": (lambda: S.compression(n_side=4), 30, 8),
    "disks_pairs": (lambda: S.suspension(n_side=13, T=0.5), 9, 4),
    "disks_three_tiles": (lambda: S.suspension(n_side=20, T=0.5), 4, 2),
    "mixed": (lambda: S.large_mixed(n_side=5, n_solvent=7001), 40, 20),
    "fan": (lambda: S.mixed_replica(3000, 0.7, 0.5, seed=4, mesh=fan(16)), 6, 3),
}


def gradients(make, steps, every, direct):
    s = F.System()
    make().replay(s)
    s.set_profiling(direct)
    s.adjoint_forward(steps, every)
    rng = np.random.Generator(np.random.PCG64(9))
    g = s.adjoint_backward(1.0, 0.5, rng.normal(size=(s.N, 2)).astype(np.float32),
                           rng.normal(size=(s.N, 2)).astype(np.float32))
    out = {k: np.array(v) for k, v in g.items()}
    s.set_profiling(False)
    out["state"] = np.stack(s.get_state())
    s.run(3)  # the exchanges of later runs go on from here
    out["later"] = np.stack(s.get_state())
    return out


@pytest.mark.parametrize("name", CASES)
def test_one_launch_equals_two_kernels_a_step(name):
    make, steps, every = CASES[name]
    a, b = gradients(make, steps, every, False), gradients(make, steps, every, True)
    assert a.keys() == b.keys()
    for k in a:
        x, y = (np.ascontiguousarray(v[k], dtype=np.asarray(v[k]).dtype) for v in (a, b))
        assert x.dtype != object and np.array_equal(x.view(np.uint8), y.view(np.uint8)), k
