"""The fast mode's large fluids with long lists run by the plain kernels, whose step
kernel is the faster one there: against direct launches bit for bit, the energies
(grouped by storage slot there, by id in the whole-run launch) among it.  At
608 tiles (four a block on 152 SMs) and with short lists the launch stays."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from test_gpu_coop import ragged_fluid

pytestmark = pytest.mark.gpu


def record(n, skin, direct):
    sc = ragged_fluid(n)
    sc.calls = [(name, (skin,) if name == "set_skin" else a) for name, a in sc.calls]
    s = F.System()
    s.set_force_mode(1)
    sc.replay(s)
    s.set_profiling(direct)
    out = []
    for steps in (1, 24):
        s.run(steps)
        out += [*s.get_state(), s.forces(), s.step_observables(), np.array([s.total_updates()])]
    s.set_profiling(False)
    return out


@pytest.mark.parametrize("n,skin,plain", [(77825, 1.5, True), (77824, 1.5, False), (77825, 0.3, False),
                                          (98304, 1.5, True)])
def test_route_by_list_length(n, skin, plain):
    a, b = (record(n, skin, direct) for direct in (False, True))
    for x, y in zip(a, b):
        if not plain and x.ndim == 2 and x.shape[1] == 6:
            x, y = x[:, 3:], y[:, 3:]
        assert np.array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8))
