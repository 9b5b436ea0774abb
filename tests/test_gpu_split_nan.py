"""FP64 passes split over four warps, on fields that hold a NaN or an infinity:
the same counters, and the same sites spoilt, as the pool's passes, which are not
split.  (A NaN staple ends the heatbath's trials at the first; it is not a link
that ran into their limit.)"""
import numpy as np
import pytest

from native import hot_fields
from su2higgs_gb300 import abi
from test_gpu_persistent import as_dict

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("content", ["fund", "adj", "su2u1s", "fundadj"])
def test_split_spoils_what_the_other_passes_spoil(content, bad):
    from su2higgs_gb300 import gpu
    p = abi.make_params(content, L=(8, 10, 6))
    f = as_dict(hot_fields(p, seed=5, phi_mean=0.5))
    f["link"][37, 1, 2] = bad
    for name in ("d0", "trip"):
        if f.get(name) is not None:
            f[name][200, 1] = bad
    lat = gpu.Lattice(p, seed=9, chain=2)
    lat.upload(**f)
    lat.run_sweeps(0, 1)
    pool = gpu.Pool(p, arena_bytes=gpu.Pool.chain_bytes(p), max_chains=1)
    pool.persistent = False
    slot = pool.add(p, seed=9, chain=2)
    pool.upload(slot, **f)
    pool.run(1)
    got, want = lat.download(), pool.download(slot)
    spoilt = 0
    for name in f:
        if f[name] is None:
            continue
        bad_sites = ~np.isfinite(want[name])
        spoilt += int(bad_sites.sum())
        assert np.array_equal(~np.isfinite(got[name]), bad_sites), name
    # at least what was put in; with a triplet no more, as a NaN action is refused
    assert spoilt >= 2
    assert np.array_equal(lat.counters()[:24], pool.counters(slot)[:24])
    pool.close()
