"""The number of a grid-wide exchange grows over the life of a context, past
2^32: runs and reverse sweeps across that number equal those of a fresh context,
bit for bit."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S
from test_gpu_coop import ragged_fluid
from test_gpu_coop_tri import fan

pytestmark = pytest.mark.gpu

SCENES = {
    "two_blocks": (lambda: ragged_fluid(129), 0),
    "every_sm": (lambda: ragged_fluid(30001), 0),
    "by_slot": (lambda: ragged_fluid(4096), 1),
    "fast": (lambda: ragged_fluid(16385), 1),
    "disks": (lambda: S.suspension(n_side=9, T=0.5), 0),
    "triangles_apart": (lambda: S.mixed_replica(3000, 0.7, 0.5, seed=4, mesh=fan(16)), 0),
}
WRAP = 1 << 32


def pair(name):
    make, mode = SCENES[name]
    out = []
    for _ in range(2):
        s = F.System()
        s.set_force_mode(mode)
        make().replay(s)
        out.append(s)
    return out


@pytest.mark.parametrize("before", [1, 2, 3, 29])
@pytest.mark.parametrize("name", SCENES)
def test_runs_across_2_to_the_32(name, before):
    s, ref = pair(name)
    s.test_set_exchanges(WRAP - before)
    for n in (1, 2, 40):
        for q in (s, ref):
            q.run(n)
        a = [*s.get_state(), s.forces(), s.step_observables(), *s.cells(), *s.neighbors()]
        b = [*ref.get_state(), ref.forces(), ref.step_observables(), *ref.cells(), *ref.neighbors()]
        for x, y in zip(a, b):
            assert np.array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8))


@pytest.mark.parametrize("name", ["every_sm", "disks"])
def test_reverse_sweep_across_2_to_the_32(name):
    grads = []
    for s, start in zip(pair(name), (None, WRAP - 25)):
        rng = np.random.Generator(np.random.PCG64(9))
        s.adjoint_forward(12, 6)
        if start:
            s.test_set_exchanges(start)
        grads.append(s.adjoint_backward(1.0, 0.5, rng.normal(size=(s.N, 2)).astype(np.float32),
                                        rng.normal(size=(s.N, 2)).astype(np.float32)))
    for k in grads[0]:
        x, y = (np.ascontiguousarray(g[k]) for g in grads)
        assert np.array_equal(x.view(np.uint8), y.view(np.uint8)), k


def test_late_timeouts_recover():
    """A bounded wait that gives up late in a context's life starts the count anew."""
    s, ref = pair("every_sm")
    pos, vel, _ = s.get_state()
    s.test_set_exchanges(WRAP + 5)
    s.test_expire_next_exchange()
    with pytest.raises(F.FemmdError):
        s.run(10)
    s.set_state(pos, vel)
    for q in (s, ref):
        q.run(10)
    for x, y in zip(s.get_state(), ref.get_state()):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
