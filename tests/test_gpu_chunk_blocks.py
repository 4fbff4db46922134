"""Persistent chunks on either side of the size from which an SM holds four of
their blocks instead of three (444 blocks of 128 spheres), against the
separate kernels of replayed graphs, bit for bit."""
import numpy as np
import pytest

from dem3d_b200 import configs
from dem3d_b200 import params as P
from dem3d_b200.system import DEMSystem

pytestmark = pytest.mark.gpu

LAST = 444 * 128  # spheres in the largest system with three blocks an SM


def _floor(n, precision):
    w = configs.settling(n=n, layer_side=48, sigma_v=3.0, euler_intervals=2, max_ncell=1 << 30,
                         precision=precision)
    return w, dict(comp=w.comp)


def _packing(n, precision):
    w = configs.dense_packing(n=n, phi=0.55, seed=1031, tile=8000)
    w.params.precision = precision
    return w, dict(radius=w.radius)


@pytest.mark.parametrize("precision", [P.PREC_FP64, P.PREC_MIXED])
@pytest.mark.parametrize("make,n", [(_floor, LAST), (_floor, LAST + 1), (_packing, 64_000)])
def test_persistent_chunks_of_either_size(make, n, precision):
    w, kind = make(n, precision)
    runs = []
    for mode in (0, 1):
        s = DEMSystem(w.params)
        s.set_launch_shape(launch_mode=mode)
        s.set_state(w.pos, w.vel, w.omega, **kind)
        s.initialize_cell_distribution()
        s.run(1, 3 + 5 * 4)
        assert mode == 0 or s.persistent_blocks() == -(-n // 128)
        runs.append((s.get_state(), s.get_contacts(), s.ncol()))
        s.close()
    (a, ca, na), (b, cb, nb) = runs
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for k in ca:
        np.testing.assert_array_equal(ca[k], cb[k], err_msg=k)
    assert na == nb and len(ca["imin"]) > 0
