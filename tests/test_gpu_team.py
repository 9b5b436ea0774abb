"""The team sweep (k_pool_team): in the automatic mode a pool whose chains are
all small sweeps each chain by a cluster of blocks, all passes of all sweeps in
one launch.  It runs the per-tile code of the other modes, so fields, counters
and sums are those of one launch per pass bit for bit -- at the edges of the
team shapes (16, 64, 128 and 256 warps of 32 sites a parity), with several
shapes at once, and with multicanonical chains whose checks reject."""
import numpy as np
import pytest

from native import hot_fields
from su2higgs_gb300 import abi
from test_gpu_persistent import as_dict, assert_same
from test_gpu_pool_muca import order_parameter, weight_around

pytestmark = pytest.mark.gpu

# half / 32 warps: < 1, 8, 16, 17 (ragged), 64, 72, 128, 144, 256: clusters of 2, 2,
# 4, 8 and 16 blocks of four warps, of 12 and 16 of eight, of 12 and 16 of sixteen
SIDES = [(2, 2, 4), (8, 8, 8), (16, 8, 8), (6, 18, 10), (16, 16, 16), (16, 16, 18), (16, 16, 32), (16, 18, 32),
         (16, 32, 32)]


@pytest.fixture(scope="module")
def gpu():
    from su2higgs_gb300 import gpu as g
    g.lib()
    return g


def make_pool(gpu, content, precision, sides, persistent):
    params = [abi.make_params(content, L=L, precision=precision, betasu2=6.0 + k) for k, L in enumerate(sides)]
    pool = gpu.Pool(params[0], arena_bytes=sum(gpu.Pool.chain_bytes(p) for p in params), max_chains=len(sides))
    pool.persistent = persistent
    slots = [pool.add(p, seed=40 + k, chain=k) for k, p in enumerate(params)]
    fields = [hot_fields(p, seed=k, phi_mean=0.5) for k, p in enumerate(params)]
    for s, f in zip(slots, fields):
        pool.upload(s, **as_dict(f))
    return pool, slots, fields


@pytest.mark.parametrize("content", ["adj", "fund", "su2u1s", "higgs2"])
@pytest.mark.parametrize("precision,sides,shapes", [(32, SIDES, 8), (32, SIDES[:3], 2), (64, SIDES[:5], 4)])
def test_team_equals_per_pass(gpu, content, precision, sides, shapes):
    a, sa, _ = make_pool(gpu, content, precision, sides, None)
    b, sb, _ = make_pool(gpu, content, precision, sides, False)
    assert a.launches_per_sweep() == shapes + 1 and not a.persistent
    for n in (1, 3):
        a.run(n)
        b.run(n)
    assert_same(a, sa, b, sb)
    ma, mb = a.measure(), b.measure()
    for x, y in zip(sa, sb):
        assert np.array_equal(ma[x], mb[y])
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_team_with_checked_chains(gpu, precision):
    sides = [(8, 8, 8), (16, 8, 8), (16, 16, 16)]
    pools = []
    for persistent in (None, False):
        pool, slots, fields = make_pool(gpu, "su2u1s", precision, sides, persistent)
        for s, f, L in zip(slots[:2], fields, sides):  # the third chain has no weight
            w = weight_around(abi.PHISQ, order_parameter(f, abi.PHISQ, L[0] * L[1] * L[2]))
            pool.muca_set(s, w.struct)
        pool.run(4)
        pools.append((pool, slots))
    (a, sa), (b, sb) = pools
    assert a.launches_per_sweep() < b.launches_per_sweep()
    assert_same(a, sa, b, sb)
    for s in sa[:2]:
        c = a.counters(s)
        assert 0 < c[abi.C_ACC_MUCA] < c[abi.C_TOTAL_MUCA]
    a.close()
    b.close()


@pytest.mark.parametrize("precision,side", [(32, (16, 32, 34)), (64, (16, 16, 18))])
def test_larger_chains_take_launches_per_pass(gpu, precision, side):
    pool, _, _ = make_pool(gpu, "adj", precision, [(8, 8, 8), side], None)
    groups = max(pool.sweep_groups[0], 1)
    assert pool.launches_per_sweep() == groups * (6 + 10 + 1)
    pool.close()
