"""The automatic choice's groups: a pool of chains too large for teams and too
small for the persistent sweep runs them in groups on several streams.  Same
kernels, so the same fields, counters and sums as one launch per pass, bit for
bit: graph and direct launches, runs of odd and even length (a group's graph is
one sweep, or two where there are many groups), chains with and without
multicanonical weights in the same groups, and a cycle of few host megabytes
cut into its own groups."""
import numpy as np
import pytest

from native import hot_fields
from su2higgs_gb300 import abi
from test_gpu_persistent import as_dict, assert_same
from test_gpu_pool_muca import order_parameter, weight_around

pytestmark = pytest.mark.gpu

SIDES = [(16, 32, 34), (8, 8, 8), (20, 24, 40), (12, 10, 6), (30, 32, 28)]


@pytest.fixture(scope="module")
def gpu():
    from su2higgs_gb300 import gpu as g
    g.lib()
    return g


def make_pool(gpu, content, precision, sides, persistent, weights=()):
    params = [abi.make_params(content, L=L, precision=precision, betasu2=6.0 + k) for k, L in enumerate(sides)]
    pool = gpu.Pool(params[0], arena_bytes=sum(gpu.Pool.chain_bytes(p) for p in params), max_chains=len(sides))
    pool.persistent = persistent
    slots = [pool.add(p, seed=70 + k, chain=k) for k, p in enumerate(params)]
    fields = [hot_fields(p, seed=k, phi_mean=0.5) for k, p in enumerate(params)]
    for k, (s, f, p) in enumerate(zip(slots, fields, params)):
        pool.upload(s, **as_dict(f))
        if k in weights:
            pool.muca_set(s, weight_around(abi.PHISQ, order_parameter(f, abi.PHISQ, p.sites())).struct)
    return pool, slots, fields


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("content,precision,weights", [("adj", 32, ()), ("fund", 64, ()), ("su2u1s", 32, (0, 3, 4))])
def test_auto_groups_equal_per_pass(gpu, content, precision, weights, graph):
    a, sa, _ = make_pool(gpu, content, precision, SIDES, None, weights)
    b, sb, _ = make_pool(gpu, content, precision, SIDES, False, weights)
    g, ns = a.sweep_groups
    assert 2 <= g <= 5 and 2 <= ns <= 4 and b.sweep_groups == (0, 1)
    for n in (1, 2, 3):
        a.run(n, graph=graph)
        b.run(n, graph=graph)
    assert_same(a, sa, b, sb)
    ma, mb = a.measure(), b.measure()
    for x, y in zip(sa, sb):
        assert np.array_equal(ma[x], mb[y])
    a.close()
    b.close()


def test_many_rounds_of_groups(gpu):
    # more than 90 MB of fields: several rounds of four groups, graphs of two sweeps
    sides = [(48, 48, 48)] * 20
    a, sa, _ = make_pool(gpu, "adj", 32, sides, None)
    b, sb, _ = make_pool(gpu, "adj", 32, sides, False)
    g, ns = a.sweep_groups
    assert g > 8 and ns == 4
    for n in (2, 3):
        a.run(n)
        b.run(n)
    assert_same(a, sa, b, sb)
    a.close()
    b.close()


def test_small_cycle_groups(gpu):
    a, sa, fields = make_pool(gpu, "fundadj", 32, SIDES * 3, None)
    b, sb, _ = make_pool(gpu, "fundadj", 32, SIDES * 3, False)
    host = [{n: np.ascontiguousarray(v) for n, v in as_dict(f).items() if v is not None} for f in fields]
    sums = a.cycle(sa, host, 3)
    b.run(3)
    mb = b.measure()
    for k, (x, y) in enumerate(zip(sa, sb)):
        want = b.download(y)
        for n in host[k]:
            assert np.array_equal(host[k][n], want[n]), (k, n)
        assert np.array_equal(sums[k], mb[y])
    a.close()
    b.close()


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("content,precision", [("adj", 32), ("fund", 32), ("su2u1s", 32), ("fund", 64)])
def test_cycle_of_many_groups(gpu, content, precision, graph, monkeypatch):
    # more than 8 groups: passes launched normally (one FP32 scalar field, no
    # U(1)) or overlapping (the others), either way the separate calls' results
    monkeypatch.setenv("SU2GPU_CYCLE_GROUPS", "10")
    sides = (SIDES * 3)[:13]
    a, sa, _ = make_pool(gpu, content, precision, sides, False)
    b, sb, fields = make_pool(gpu, content, precision, sides, None)
    want = [{k: np.ascontiguousarray(v) for k, v in as_dict(f).items() if v is not None} for f in fields]
    got = [{k: v.copy() for k, v in f.items()} for f in want]
    for _ in range(2):
        a.upload_many(sa, want)
        a.run(2, graph=graph)
        ma = a.measure()
        a.download_many(sa, want)
        mb = b.cycle(sb, got, 2, graph=graph)
        for j, s in enumerate(sa):
            assert np.array_equal(mb[j], ma[s])
            assert all(np.array_equal(got[j][k], want[j][k]) for k in want[j])
    assert all(np.array_equal(a.counters(x), b.counters(y)) for x, y in zip(sa, sb))
    a.close()
    b.close()
