"""Candidate rows and the relink at the edges of their variants, bit for bit
against the oracle: the largest system whose relink and rows share a launch
and the smallest whose do not, more movers than a pass records, cells whose
lists do not fit their slots, and rows so long that a warp tests them in
several windows."""
import numpy as np
import pytest

from dem3d_b200 import configs
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
