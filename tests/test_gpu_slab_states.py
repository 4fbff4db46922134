"""A slab's context takes a state of more particles than the one it was made
with: its ghost stamps and particle lists grow with it, and the composed run
equals the undivided one bit for bit."""
import numpy as np
import pytest

from dem3d_b200 import params as P
from dem3d_b200 import slab as S
from dem3d_b200.system import DEMSystem
from tests.test_gpu_scale import transfer
from tests.test_gpu_slab import _base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("again", [False, True])
def test_slab_takes_a_larger_state(again):
    w, g = _base(P.PREC_FP64)
    ref = DEMSystem(w.params)
    transfer(g, ref, radius=w.radius)
    slabs = []
    for z0, z1 in S.slab_ranges(g.grid()[2], 2):
        s = DEMSystem(w.params)
        s.set_state(w.pos[:500], w.vel[:500], w.omega[:500], radius=w.radius[:500])
        s.initialize_cell_distribution()
        s.slab_set_range(z0, z1)
        transfer(g, s, radius=w.radius)
        if again:
            s.slab_set_range(z0, z1)
        slabs.append(s)
    tr = S.LocalTransport(slabs, periodic=True, cap_bytes=64 << 20)
    for step in range(21, 33):
        S.move_particles(tr, step)
    ref.run(21, 32)
    want, got = ref.get_state(), S.compose_state(slabs)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
