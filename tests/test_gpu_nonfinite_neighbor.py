"""A non-finite position in the reference-exact mode: its pairs are outside every
cutoff (the comparison is false), so its neighbours go on undisturbed and the
state that a failed run leaves behind shows the one particle.  Runs of a few
steps, before a rebuild could meet the position.

Cases: single systems as one launch and by direct launches, a system beyond the
whole-run launch, one and two types, walls, and the batched replicas; an
infinite or NaN coordinate in the start state (stale lists) and a NaN velocity
(the position of the first drift)."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from test_gpu_coop import ragged_fluid

pytestmark = pytest.mark.gpu
BAD = 1234

SCENES = {
    "fluid": lambda: ragged_fluid(2300),
    "two_types": lambda: ragged_fluid(2300, types=2),
    "walls": lambda: ragged_fluid(2300, density=0.6, pbc=0),
    "large": lambda: ragged_fluid(120001),
}


def spoiled(pos, vel, what):
    pos, vel = pos.copy(), vel.copy()
    if what == "velocity":
        vel[BAD] = np.nan
    else:
        pos[BAD, 1] = {"nan": np.nan, "inf": np.inf, "-inf": -np.inf}[what]
    return pos, vel


def check(s, pos):
    x, v, a = s.get_state()
    rows = ~(np.isfinite(x).all(1) & np.isfinite(v).all(1) & np.isfinite(a).all(1))
    assert rows[BAD] and rows.sum() == 1
    # a neighbour was there to be disturbed
    d = np.linalg.norm(np.delete(pos, BAD, 0) - pos[BAD], axis=1)
    assert d.min() < 2.5


@pytest.mark.parametrize("what", ["nan", "inf", "-inf", "velocity"])
@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("name", SCENES)
def test_only_the_particle_itself(name, direct, what):
    s = F.System()
    SCENES[name]().replay(s)
    s.run(2)
    pos, vel, _ = s.get_state()
    s.set_state(*spoiled(pos, vel, what))
    s.set_profiling(direct)
    with pytest.raises(F.FemmdError):
        s.run(3)
    check(s, pos)


@pytest.mark.parametrize("what", ["nan", "inf", "-inf", "velocity"])
@pytest.mark.parametrize("types", [1, 2])
def test_batched_replicas(types, what):
    b, systems = F.Batch(0), []
    for k in range(3):
        s = F.System()
        ragged_fluid(2300 + k, types=types, seed=k).replay(s)
        systems.append(s)
        b.add(s)
    b.run(2)
    pos, vel, _ = systems[1].get_state()
    systems[1].set_state(*spoiled(pos, vel, what))
    if what == "velocity":
        b.run(3)  # the batch flags forces and positions: this one shows at the next rebuild
    else:
        with pytest.raises(F.FemmdError):
            b.run(3)
    check(systems[1], pos)
    for k in (0, 2):
        assert all(np.isfinite(x).all() for x in systems[k].get_state())
