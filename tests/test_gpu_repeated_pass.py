"""A pass that stops for room (here: longer candidate rows) and is repeated
sees the walls and the clock of its step, not those that the launch it stopped
in would have had: before the first step of a launch, and for steps that are
not numbered on from the last one, the walls are not those of (step - 1)*dt."""
import numpy as np
import pytest

from dem3d_b200 import configs
from dem3d_b200 import params as P
from dem3d_b200.system import DEMSystem
from tests.oracle_lib import oracle_system

pytestmark = pytest.mark.gpu


def _bed(make, n, order):
    """Two sizes of spheres lying on a floor that shakes, between four walls."""
    w = configs.bidisperse_settling(n=n, width=24.0, headroom=6.0, sigma_v=1.0,
                                    method_order=order, euler_intervals=7)
    w.params.walls[0].position[2] += 0.05  # (the lowest spheres are 0.02 and 0.03 above it)
    s = make(w.params)
    s.set_particle_removal(False)
    s.set_state(w.pos, w.vel, w.omega, comp=w.comp)
    motions = [P.wall_motion(tuple(w.params.walls[j].position), (0.0,) * 3, (0.0,) * 3, (0.0,) * 3)
               for j in range(w.params.n_walls)]
    z = w.params.walls[0].position[2]
    motions[0] = P.wall_motion((0.0, 0.0, z), (0.0, 0.0, 0.1), (0.0, 0.0, 20.0),
                               (0.0, 0.0, 0.25))
    s.set_wall_motion(motions)
    s.initialize_cell_distribution()
    return s


def _call(step):
    return lambda s: s.move_particles(step)


def _run(first, last):
    return lambda s: s.run(first, last)


# name: spheres, method order, the calls before, the call whose pass stops,
# the calls after it
CASES = {
    "first_call": (1500, 1, [], _call(1), [_call(2)]),
    "renumbered_call": (1500, 4, [_run(1, 4)], _call(100), [_call(101)]),
    "call_after_the_start_up": (1500, 4, [_run(1, 3)], _call(4), [_run(5, 12)]),
    "cluster_after_the_start_up": (1500, 4, [_run(1, 3)], _run(4, 20), [_run(21, 30)]),
    "cluster_from_rest": (1500, 1, [], _run(1, 20), [_run(21, 30)]),
    "graph_after_the_start_up": (3000, 4, [_run(1, 3)], _run(4, 20), [_run(21, 30)]),
    "graph_from_rest": (3000, 1, [], _run(1, 20), [_run(21, 30)]),
}


@pytest.mark.parametrize("name", CASES)
def test_walls_of_a_repeated_pass(name):
    n, order, before, stop, after = CASES[name]
    g, o = _bed(DEMSystem, n, order), _bed(oracle_system, n, order)
    for call in before:
        for s in (g, o):
            call(s)
    assert g.row_stats()["row_capacity"] == 32
    g.set_tuning(0.5, 0)  # rows of more than 32 candidates from the next pass on
    for call in [stop, *after]:
        for s in (g, o):
            call(s)
        assert g.row_stats()["row_capacity"] > 32
        a, b = g.get_state(), o.get_state()
        for k in b:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
        ca, cb = g.get_contacts(), o.get_contacts()
        for k in cb:
            np.testing.assert_array_equal(ca[k], cb[k], err_msg=k)
        wa, wb = g.walls(), o.walls()
        for k in wb:
            np.testing.assert_array_equal(wa[k], wb[k], err_msg=k)
        if call is stop:  # the floor is touched in the repeated pass
            assert np.count_nonzero(ca["iw"] == 0) > 0
    g.close()
    o.close()
