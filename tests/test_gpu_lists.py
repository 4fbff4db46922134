"""Relink and rows as one cluster's launch (calls of their own) and as two
kernels (captured chunks), one after the other on the same system, with many
spheres changing cell in every pass: bit for bit against the oracle."""
import numpy as np
import pytest

from dem3d_b200 import configs
from dem3d_b200 import params as P
from dem3d_b200.system import DEMSystem
from tests.oracle_lib import oracle_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2049, 16384, 16385])
def test_merged_and_separate_lists(n):
    w = configs.settling(n=n, layer_side=32, sigma_v=60.0, euler_intervals=2,
                         max_ncell=1 << 30, first_height=1.0, precision=P.PREC_FP64)
    g, o = DEMSystem(w.params), oracle_system(w.params)
    for s in (g, o):
        s.set_particle_removal(False)
        s.set_state(w.pos, w.vel, w.omega, comp=w.comp)
        s.initialize_cell_distribution()
        s.run(1, 7)
    before = g.launch_count()
    for step in range(8, 12):
        g.move_particles(step)
    per_call = (g.launch_count() - before) / 4
    before = g.launch_count()
    g.run(12, 19)
    per_step = (g.launch_count() - before) / 8
    assert per_call == (8 if n <= 16384 else 10) and per_step == 10
    o.run(8, 19)
    a, b = g.get_state(), o.get_state()
    for k in b:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for x, y, k in zip(g.get_cells(), o.get_cells(), ("cell", "order", "start")):
        np.testing.assert_array_equal(x, y, err_msg=k)
    ca, cb = g.get_contacts(), o.get_contacts()
    for k in cb:
        np.testing.assert_array_equal(ca[k], cb[k], err_msg=k)
    assert g.ncol() == o.ncol() > 0
