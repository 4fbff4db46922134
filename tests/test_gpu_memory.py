"""Growing an array when the device's memory is used up: the call reports it,
the calls after it refuse to run on what is left, the particles can still be
read, and a new state runs as in a new context."""
import numpy as np
import pytest

from dem3d_b200 import configs
from dem3d_b200.system import DEMError, DEMSystem

pytestmark = pytest.mark.gpu


def _fill(torch):
    """All device memory but 16 MB at the most."""
    torch.cuda.empty_cache()
    hold = []
    for size in (8 << 30, 1 << 30, 128 << 20, 10 << 20):
        while torch.cuda.mem_get_info()[0] > size + (6 << 20):
            try:
                hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                break
    return hold


def _set(s, w):
    s.set_state(w.pos, w.vel, w.omega, comp=w.comp)
    s.initialize_cell_distribution()


@pytest.mark.parametrize("reorder", [0, 4])
def test_rows_that_find_no_memory(reorder):
    import torch
    # 51 MB of rows, 77 MB at the least when they grow
    w = configs.bidisperse_settling(n=400_000, width=96.0, headroom=6.0, sigma_v=1.0, euler_intervals=2)
    g = DEMSystem(w.params)
    g.set_particle_removal(False)
    g.set_reorder(reorder)
    _set(g, w)
    g.run(1, 11)
    kept = g.get_state()
    g.run(12, 15)
    g.set_tuning(0.5, 0)  # rows of more than 32 candidates
    hold = _fill(torch)
    with pytest.raises(DEMError, match="out of memory"):
        g.run(16, 30)
    for call in (lambda: g.run(16, 30), lambda: g.move_particles(16), g.compute_accelerations,
                 g.get_cells):
        with pytest.raises(DEMError):
            call()
    if reorder:  # (the storage cannot go back into order without room, either)
        del hold
        torch.cuda.empty_cache()
    got = g.get_state()
    assert np.isfinite(got["pos"]).all()
    assert np.abs(got["pos"] - kept["pos"]).max() < 1.0
    g.initialize_cell_distribution()
    with pytest.raises(DEMError, match="set the state again"):
        g.run(16, 30)
    hold = None
    torch.cuda.empty_cache()
    _set(g, w)
    g.run(1, 15)
    assert g.row_stats()["row_capacity"] > 32
    ref = DEMSystem(w.params)
    ref.set_particle_removal(False)
    ref.set_tuning(0.5, 0)
    _set(ref, w)
    ref.run(1, 15)
    a, b = g.get_state(), ref.get_state()
    for k in b:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    g.close()
    ref.close()


def test_a_state_that_finds_no_memory():
    import torch
    w = configs.settling(n=400_000, layer_side=100, euler_intervals=2, max_ncell=1 << 30)
    few = slice(0, 500)
    g = DEMSystem(w.params)
    g.set_state(w.pos[few], w.vel[few], w.omega[few], comp=w.comp[few])
    g.initialize_cell_distribution()
    g.run(1, 8)
    hold = _fill(torch)
    with pytest.raises(DEMError, match="out of memory"):
        _set(g, w)
    for call in (g.get_state, g.initialize_cell_distribution, lambda: g.run(9, 12)):
        with pytest.raises(DEMError, match="state"):
            call()
    del hold
    torch.cuda.empty_cache()
    _set(g, w)
    g.run(1, 8)
    assert np.isfinite(g.get_state()["pos"]).all()
    g.close()
