"""The ABM ring at every method order, for each way dem_run launches its steps:
a cluster launch of a small system, replayed graphs, persistent chunks, and the
separate kernels one by one (kernel profiling on).  The ring holds order - 1
past steps and a spare slot, so its rotation comes back after as many steps as
the order: a launch of several steps must follow it.  Bit for bit against the
separate kernels, and in FP64 against the oracle."""
import numpy as np
import pytest

from dem3d_b200 import configs
from dem3d_b200 import params as P
from dem3d_b200.system import DEMSystem
from tests.oracle_lib import oracle_system

pytestmark = pytest.mark.gpu

PRECISIONS = [P.PREC_FP64, P.PREC_MIXED]


def _bed(make, n, order, precision, moving):
    w = configs.settling(n=n, layer_side=12, sigma_v=3.0, euler_intervals=2, max_ncell=1 << 30,
                         method_order=order, precision=precision)
    s = make(w.params)
    s.set_state(w.pos, w.vel, w.omega, comp=w.comp)
    if moving:
        z = w.params.walls[0].position[2]
        s.set_wall_motion([P.wall_motion((0.0, 0.0, z), (0.0, 0.0, 0.05), (0.0, 0.0, 20.0),
                                         (0.0, 0.0, 0.25))])
    s.initialize_cell_distribution()
    return s


def _hopper(make, precision):
    w = configs.hopper(n=600, seed=1005)
    w.params.precision = precision
    s = make(w.params)
    s.set_state(w.pos, w.vel, w.omega, comp=w.comp, radius=w.radius)
    s.initialize_cell_distribution()
    return s


def _same(a, b):
    assert a.n == b.n
    x, y = a.get_state(), b.get_state()
    for k in x:
        np.testing.assert_array_equal(x[k], y[k], err_msg=k)
    if a.nprev > 0:
        np.testing.assert_array_equal(a.logical_ring(), b.logical_ring(), err_msg="ring")
    x, y = a.get_contacts(), b.get_contacts()
    for k in x:
        np.testing.assert_array_equal(x[k], y[k], err_msg=k)
    np.testing.assert_array_equal(a.walls()["position"], b.walls()["position"])
    assert a.ncol() == b.ncol()


def _launches(s, first, last):
    before = s.launch_count()
    s.run(first, last)
    return s.launch_count() - before


# 41 steps in three calls: more than a cluster launch holds, then one step and
# a remainder from whatever rotation the ring is left in
PARTS = ((5, 37), (38, 38), (39, 45))


def _follow(a, others, launches):
    """`a` by its launches (at most so many per step), `others` beside it."""
    for s in (a, *others):
        s.run(1, 4)
    for first, last in PARTS:
        assert _launches(a, first, last) <= launches * (last - first + 1)
        for s in others:
            s.run(first, last)
        for s in others:
            _same(a, s)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_cluster_launches(order, precision):
    def make(m):
        return _bed(m, 333, order, precision, True)
    a, b = make(DEMSystem), make(DEMSystem)
    b.set_profiling(True)
    others = [b] if precision else [b, make(oracle_system)]
    _follow(a, others, 1)
    assert a.ncol() > 0


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("mode", [0, 1])
def test_graphs_and_persistent_chunks(mode, order, precision):
    def make(m):
        return _bed(m, 2049, order, precision, False)
    a, b = make(DEMSystem), make(DEMSystem)
    a.set_launch_shape(launch_mode=mode)
    b.set_profiling(True)
    others = [b] if precision else [b, make(oracle_system)]
    _follow(a, others, 10)
    assert mode == 0 or a.persistent_blocks() > 0
    assert a.ncol() > 0


def test_cluster_and_separate_kernels_agree_on_a_cone_in_mixed_precision():
    a, b = _hopper(DEMSystem, P.PREC_MIXED), _hopper(DEMSystem, P.PREC_MIXED)
    b.set_profiling(True)
    for s in (a, b):
        s.run(1, 700)
    steps = _launches(a, 701, 800), _launches(b, 701, 800)
    assert steps[0] <= 100 and steps[1] >= 800
    _same(a, b)
    assert np.count_nonzero(a.get_contacts()["iw"] == 0) > 0  # the cone is touched
