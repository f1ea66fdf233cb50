"""The backward pass's recomputation of a segment by the kernels of the forward
runs: with property averaging, or with the profiling switched between the two
passes, and in systems whose cells are too crowded for the whole-run launch.
The gradients are those of a plain forward and backward pass, bit for bit."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from test_gpu_coop import ragged_fluid
from test_gpu_coop_left import CELL_CAP, most_per_cell, small_particles

pytestmark = pytest.mark.gpu

SCENES = {
    "fluid": lambda: ragged_fluid(2300),
    "crowded": lambda: small_particles(45, 0.4472, 0.4, 0.0, 0.002)[0],
}


def gradients(make, forward, backward):
    """forward, backward: 'whole', 'direct' (profiling) or 'average'."""
    s = F.System()
    make().replay(s)

    def switch(how):
        s.set_profiling(how == "direct")
        s.set_property_averaging(how == "average", 1000, 1000)

    switch(forward)
    s.adjoint_forward(30, 10)
    switch(backward)
    rng = np.random.Generator(np.random.PCG64(9))
    g = s.adjoint_backward(1.0, 0.5, rng.normal(size=(s.N, 2)).astype(np.float32),
                           rng.normal(size=(s.N, 2)).astype(np.float32))
    out = {k: np.array(v) for k, v in g.items()}
    switch("whole")
    out["state"] = np.stack(s.get_state())
    s.run(3)
    out["later"] = np.stack(s.get_state())
    return out


@pytest.mark.parametrize("forward,backward", [("average", "average"), ("average", "whole"), ("direct", "whole"),
                                              ("whole", "direct"), ("whole", "whole")])
@pytest.mark.parametrize("name", SCENES)
def test_recomputation_routes(name, forward, backward):
    make = SCENES[name]
    if name == "crowded":
        sc, box = small_particles(45, 0.4472, 0.4, 0.0, 0.002)
        s = F.System()
        sc.replay(s)
        assert most_per_cell(s.get_state()[0], box) > CELL_CAP
    a, b = gradients(make, forward, backward), gradients(make, "direct", "direct")
    assert a.keys() == b.keys()
    for k in a:
        x, y = np.ascontiguousarray(a[k]), np.ascontiguousarray(b[k])
        assert x.dtype != object and np.array_equal(x.view(np.uint8), y.view(np.uint8)), k
