"""Two doublets in FP64 on both sides of the line where passes stop being split
over four warps (384 blocks of 32 sites of a parity), one sweep against the
oracle.  The overrelaxation of two doublets is the least well conditioned of the
updates: over 40 configurations of these sizes, with passes split or not, its
largest distance from the oracle was 2.5e-11, so fields have to agree to 1e-10
here (an update of the wrong sites or with the wrong uniforms is off by 0.1 and
more); the counters, which any other decision would move, have to be equal."""
import numpy as np
import pytest

from native import Oracle, hot_fields
from su2higgs_gb300 import abi
from test_gpu_parity import max_diff, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [23, 24, 25])
@pytest.mark.parametrize("L", [(32, 32, 24), (28, 40, 22)])
def test_two_doublets_at_the_line(L, seed):
    from su2higgs_gb300 import gpu
    p = abi.make_params("higgs2", L=L)
    f = hot_fields(p, seed=seed, phi_mean=0.5)
    lat = gpu.Lattice(p, seed=seed + 8)
    upload(lat, f)
    o = Oracle(p)
    o.put(f)
    lat.update_lattice(3)
    o.set_rng(seed + 8, 3)
    o.update()
    for k, v in max_diff(lat.download(), o.get()).items():
        assert v < 1e-10, (k, v)
    assert np.array_equal(lat.counters()[:22], o.counters()[:22])
