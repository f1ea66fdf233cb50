"""A grid-wide exchange of the reverse sweep that gives up (block 0 withholds its
record) ends the backward pass with FEMMD_TIMEOUT; the context then runs, and
differentiates, like a fresh one.  With property averaging on, the segments are
recomputed by the plain kernels and the sweep's is the first exchange."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S
from test_gpu_coop import ragged_fluid

pytestmark = pytest.mark.gpu
SCENES = {"fluid": lambda: ragged_fluid(4001), "disks": lambda: S.suspension(n_side=5, T=0.5)}


def gradients(s):
    rng = np.random.Generator(np.random.PCG64(9))
    return s.adjoint_backward(1.0, 0.5, rng.normal(size=(s.N, 2)).astype(np.float32),
                              rng.normal(size=(s.N, 2)).astype(np.float32))


@pytest.mark.parametrize("name", SCENES)
def test_expired_sweep_reports_and_recovers(name):
    s, ref = F.System(), F.System()
    for q in (s, ref):
        SCENES[name]().replay(q)
    pos, vel, _ = s.get_state()
    s.set_property_averaging(True, 1000, 1000)
    s.adjoint_forward(12, 4)
    s.test_expire_next_exchange()
    with pytest.raises(F.FemmdError) as e:
        gradients(s)
    assert "expired" in str(e.value)
    s.set_property_averaging(False)
    s.set_state(pos, vel)
    ref.set_state(pos, vel)
    for q in (s, ref):
        q.adjoint_forward(12, 4)
    a, b = gradients(s), gradients(ref)
    for k in a:
        x, y = np.ascontiguousarray(a[k]), np.ascontiguousarray(b[k])
        assert np.array_equal(x.view(np.uint8), y.view(np.uint8)), k
    for x, y in zip(s.get_state(), ref.get_state()):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
