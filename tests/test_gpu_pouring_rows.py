"""Pouring after the candidate rows have grown: rows that grow while few
spheres are in must have room for every sphere that is still to be poured
(a row entry k of sphere p lies at k*n + p, and n rises)."""
import numpy as np
import pytest

from dem3d_b200 import _abi, configs
from dem3d_b200 import params as P
from dem3d_b200.system import DEMSystem
from tests.oracle_lib import oracle_system

pytestmark = pytest.mark.gpu


def crowded_box():
    """Two spheres of diameter 3 within 125 of diameter 1, and as many small
    ones poured from the top."""
    L, lz = 14.0, 16.0
    lattice = np.stack(np.meshgrid(*[np.arange(6) - 2.5] * 3, indexing="ij"), -1).reshape(-1, 3)
    large = np.array([(-1.5, -1.5, -1.5), (1.5, 1.5, 1.5)])
    far = (np.linalg.norm(lattice[:, None] - large[None], axis=2) > 2.0).all(1)
    small = 1.001 * lattice[far]
    pos = np.concatenate([small, large]) - (0.0, 0.0, 0.5 * lz - 4.0)
    comp = np.array([0] * len(small) + [1] * 2, np.int32)
    walls = [P.rectangle((0.0, 0.0, -0.5 * lz), 0.5 * L, 0.5 * L,
                         stiffness=2.0 * configs.KN, shear_stiffness=2.0 * configs.KT)]
    comps = [P.Component(len(small), 1.0, configs.DENSITY, 2.0 * configs.KN, 2.0 * configs.KT),
             P.Component(2, 3.0, configs.DENSITY, 2.0 * configs.KN, 2.0 * configs.KT)]
    prm, _ = P.component_params(comps, walls, [[0.7] * 2] * 2, [[0.7] * 2] * 2, [[0.5] * 2] * 2,
                                [[0.7]] * 2, [[0.7]] * 2, [[0.5]] * 2, lbox=(L, L, lz),
                                pbc=(True, True, False), gravity=(0.0, 0.0, -10.0),
                                time_step=5e-4, method_order=4, euler_intervals=4)
    pour = P.pouring([3 * len(small), 2], _abi.POUR_RECTANGLE, (13.0, 13.0), 30, 2 * 5e-4, 5e-4)
    pour.velocity_z = -40.0
    return prm, pos, comp, pour


def start(make, prm, pos, comp, pour):
    s = make(prm)
    s.set_pouring(pour)  # (before the state: the arrays are laid out for the targets)
    s.set_state(pos, np.zeros_like(pos), np.zeros_like(pos), comp=comp)
    s.initialize_cell_distribution()
    s.set_rng(dummy=-7)
    return s


@pytest.mark.parametrize("precision", [P.PREC_FP64, P.PREC_MIXED])
def test_rows_grown_before_pouring(precision):
    prm, pos, comp, pour = crowded_box()
    prm.precision = precision
    g = start(DEMSystem, prm, pos, comp, pour)
    g.set_tuning(0.5, 0)  # (a skin of 1.5: a large sphere's row holds about 60)
    g.set_pouring(None)
    g.run(1, 8)
    grown = g.row_stats()["row_capacity"]
    assert grown > 32 and g.n == len(pos)
    g.set_pouring(pour)
    g.run(9, 2600)
    assert g.row_stats()["row_capacity"] == grown  # (no later growth hid the first)
    assert grown * len(pos) < 25 * g.n
    if precision == P.PREC_MIXED:
        assert np.isfinite(g.get_state()["pos"]).all()
        return
    o = start(oracle_system, prm, pos, comp, pour)
    o.set_pouring(None)
    o.run(1, 8)
    o.set_pouring(pour)
    o.run(9, 2600)
    assert g.n == o.n
    a, b = g.get_state(), o.get_state()
    for k in b:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    ca, cb = g.get_contacts(), o.get_contacts()
    for k in cb:
        np.testing.assert_array_equal(ca[k], cb[k], err_msg=k)
    assert g.rng() == o.rng() and g.ncol() == o.ncol()
