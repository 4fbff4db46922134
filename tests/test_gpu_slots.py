"""The slots that hold each cell's list: half as many where the full number
would take much of the free memory (a wide, mostly empty grid), with the same
trajectory.  A list past the slots is walked link by link."""
import numpy as np
import pytest

from dem3d_b200 import configs
from dem3d_b200.system import DEMSystem
from tests.oracle_lib import oracle_system

pytestmark = pytest.mark.gpu


def _run(make, w):
    s = make(w.params)
    s.set_particle_removal(False)
    s.set_state(w.pos, w.vel, w.omega, comp=w.comp)
    s.initialize_cell_distribution()
    return s


def test_half_the_slots_where_memory_is_short():
    import torch
    # 7 x 7 cells of 3.41 x 3.41 x 3.0 per layer: about 34 small spheres each
    w = configs.bidisperse_settling(n=1500, width=23.9, headroom=65000.0, sigma_v=100.0,
                                    euler_intervals=2)
    gib, used, systems = 1 << 30, [], []
    for fill in (True, False):
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        hold = torch.empty(free - 3 * gib // 2 if fill else 1, dtype=torch.uint8, device="cuda")
        before = torch.cuda.mem_get_info()[0]
        systems.append(_run(DEMSystem, w))
        used.append(before - torch.cuda.mem_get_info()[0])
        del hold
    torch.cuda.empty_cache()
    ncell = int(np.prod(systems[0].grid()))
    assert ncell * 256 > 3 * gib // 16
    assert used[1] - used[0] > 120 * ncell  # 32 slots of 4 bytes more
    o = _run(oracle_system, w)
    longest = np.bincount(o.get_cells()[0]).max()
    assert 32 < longest <= 64
    for s in (*systems, o):
        s.run(1, 40)
    b, cb = o.get_state(), o.get_contacts()
    for s in systems:
        a, ca = s.get_state(), s.get_contacts()
        for k in b:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
        for k in cb:
            np.testing.assert_array_equal(ca[k], cb[k], err_msg=k)
        for x, y in zip(s.get_cells(), o.get_cells()):
            np.testing.assert_array_equal(x, y)
        assert s.ncol() == o.ncol() > 0
        s.close()
    o.close()
