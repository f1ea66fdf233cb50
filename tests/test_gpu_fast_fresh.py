"""Fast mode, bonded particles: a context whose first run is a whole-run launch has
no cell-ordered mirror of the positions yet.  Drifts on their own (do_step, a
trajectory frame inside the first run), which write the mirror, follow it here; the results are those of the plain kernels (direct
launches) bit for bit, as the arithmetic is the same."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S

pytestmark = pytest.mark.gpu


def record(direct, path):
    s = F.System()
    s.set_force_mode(1)
    S.large_mixed(n_side=5, n_solvent=7001).replay(s)
    if path:
        s.set_trajectory(path, 3)
    s.set_profiling(direct)
    s.run(7)
    out = [*s.get_state(), s.forces()]
    for _ in range(4):
        s.do_step()
    out += [*s.get_state(), s.forces()]
    s.run(9)
    s.do_step()
    out += [*s.get_state(), s.forces(), np.array([s.steps()])]
    return out


@pytest.mark.parametrize("frames", [False, True])
def test_drifts_after_a_first_whole_run(frames, tmp_path):
    a = record(False, tmp_path / "a.vtf" if frames else None)
    b = record(True, tmp_path / "b.vtf" if frames else None)
    for x, y in zip(a, b):
        assert np.array_equal(np.ascontiguousarray(x).view(np.uint8), np.ascontiguousarray(y).view(np.uint8))
