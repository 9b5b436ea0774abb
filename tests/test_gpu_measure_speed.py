"""Measurements of the contents that have no kernels of their own (two doublets,
doublet and triplet) keep pace: ratios of times on the same GPU, with lines
half-way between what such a measurement takes and what it took when its sites'
loop and its block sums were the slow part."""
import time

import numpy as np
import pytest

from native import hot_fields
from su2higgs_gb300 import abi
from test_gpu_persistent import as_dict

pytestmark = pytest.mark.gpu


def best_time(measure):
    t = []
    for _ in range(30):
        t0 = time.perf_counter()
        measure()
        t.append(time.perf_counter() - t0)
    return min(t)


def test_two_doublets_of_128():
    # 8 times the sites, a quarter of them in parallel: 4.1 (256 against 66 us); it was 7.7
    from su2higgs_gb300 import gpu
    best = []
    for side in (64, 128):
        lat = gpu.Lattice(abi.make_params("higgs2", L=(side,) * 3, precision=32), seed=1)
        lat.run_sweeps(0, 1)
        best.append(best_time(lat.measure))
        lat.close()
    assert best[1] < 5.8 * best[0], best


def test_pool_of_small_chains():
    # one triplet against doublet and triplet, 150 chains: 1.13 (122, 138 us); it was 1.7
    from su2higgs_gb300 import gpu
    best = []
    for content in ("adj", "fundadj"):
        params = [abi.make_params(content, L=((12, 16)[k % 2],) * 3, precision=32) for k in range(150)]
        pool = gpu.Pool(params[0], arena_bytes=sum(gpu.Pool.chain_bytes(p) for p in params), max_chains=len(params))
        slots = [pool.add(p, seed=k, chain=k) for k, p in enumerate(params)]
        fields = [as_dict(hot_fields(p, seed=1, phi_mean=0.5)) for p in params[:2]]
        pool.upload_many(slots, [{n: np.ascontiguousarray(a) for n, a in fields[k % 2].items() if a is not None}
                                 for k in range(len(slots))])
        pool.run(1)
        best.append(best_time(pool.measure))
        pool.close()
    assert best[1] < 1.4 * best[0], best
