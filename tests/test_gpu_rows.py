"""Candidate rows and the relink at the edges of their variants, bit for bit
against the oracle: the largest system whose relink and rows share a launch
and the smallest whose do not, more movers than a pass records, cells whose
lists do not fit their slots, and rows so long that a warp tests them in
several windows."""
import numpy as np
import pytest

from dem3d_b200 import configs
from dem3d_b200 import params as P
from dem3d_b200.system import DEMSystem
from tests.oracle_lib import oracle_system

pytestmark = pytest.mark.gpu


def _settling(n, sigma_v):
    return configs.settling(n=n, layer_side=32, sigma_v=sigma_v, euler_intervals=2,
                            max_ncell=1 << 30, first_height=1.0)


CASES = {
    "merged_most": (lambda: _settling(16384, 60.0), 0.05, 20),
    "separate_least": (lambda: _settling(16385, 60.0), 0.05, 20),
    "movers_past_the_record": (lambda: _settling(16385, 600.0), 0.05, 8),
    "lists_past_the_slots": (lambda: configs.bidisperse_settling(
        n=3000, width=24.0, headroom=6.0, sigma_v=100.0, euler_intervals=4, max_ncell=64),
        0.05, 40),
    "windows": (lambda: configs.bidisperse_settling(
        n=6000, width=24.0, headroom=6.0, sigma_v=100.0, euler_intervals=4), 0.5, 40),
}


@pytest.mark.parametrize("name", CASES)
def test_rows_follow_the_oracle(name):
    make, skin, steps = CASES[name]
    w = make()
    g, o = DEMSystem(w.params), oracle_system(w.params)
    g.set_tuning(skin, 0)
    for s in (g, o):
        s.set_particle_removal(False)
        s.set_state(w.pos, w.vel, w.omega, comp=w.comp, radius=w.radius)
        s.initialize_cell_distribution()
        s.run(1, steps)
    a, b = g.get_state(), o.get_state()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for x, y, k in zip(g.get_cells(), o.get_cells(), ("cell", "order", "start")):
        np.testing.assert_array_equal(x, y, err_msg=k)
    ca, cb = g.get_contacts(), o.get_contacts()
    for k in ca:
        np.testing.assert_array_equal(ca[k], cb[k], err_msg=k)
    assert g.ncol() == o.ncol() > 0
    g.close()
    o.close()


@pytest.mark.parametrize("n,precision", [(1, 0), (127, 0), (2047, 0), (2048, 1), (2049, 0)])
def test_cluster_steps_equal_single_calls(n, precision):
    """The largest systems whose steps are one cluster launch and the smallest
    past them: runs of 33 and 1 steps (a full launch and a remainder), with a
    moving floor, against one call per step; FP64 against the oracle too."""
    def make(factory):
        w = configs.settling(n=n, layer_side=12, sigma_v=3.0, euler_intervals=2,
                             max_ncell=1 << 30)
        w.params.precision = precision
        s = factory(w.params)
        s.set_state(w.pos, w.vel, w.omega, comp=w.comp)
        z = w.params.walls[0].position[2]
        s.set_wall_motion([P.wall_motion((0.0, 0.0, z), (0.0, 0.0, 0.05), (0.0, 0.0, 20.0),
                                         (0.0, 0.0, 0.25))])
        s.initialize_cell_distribution()
        return s
    a, b = make(DEMSystem), make(DEMSystem)
    a.run(1, 36)
    a.run(37, 37)
    b.run(1, 3)
    for k in range(4, 38):
        b.move_particles(k)
    other = [b] if precision else [b, make(oracle_system)]
    if not precision:
        other[1].run(1, 37)
    for o in other:
        x, y = a.get_state(), o.get_state()
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)
        assert a.ncol() == o.ncol()
        np.testing.assert_array_equal(a.walls()["position"], o.walls()["position"])
