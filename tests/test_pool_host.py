"""Host code of the pool's grouped sweep, on a CUDA runtime that runs nothing
(fake_gpu.py): what it enqueues where, and what it leaves behind when a call
fails."""
import numpy as np
import pytest

from fake_gpu import fake_gpu
from su2higgs_gb300 import abi

SIDES = [(16, 32, 34), (20, 24, 40), (30, 32, 28), (24, 28, 30), (26, 26, 26)]


@pytest.fixture
def env(monkeypatch, tmp_path_factory):
    return fake_gpu(monkeypatch, tmp_path_factory.getbasetemp())


def make_pool(gpu, sides=SIDES, **kw):
    params = [abi.make_params("adj", L=L, **{"precision": 32, **kw}) for L in sides]
    pool = gpu.Pool(params[0], arena_bytes=sum(gpu.Pool.chain_bytes(p) for p in params), max_chains=len(sides))
    for k, p in enumerate(params):
        pool.add(p, seed=k, chain=k)
    return pool


def forked_and_joined(ops):
    """(streams with work that other streams' calls wait for, streams joined):
    a stream is forked once it waits for an event of the pool's stream and
    joined when the pool's stream waits for an event recorded on it last."""
    records, worked, home = {}, {}, None
    joined = set()
    for what, a, b in ops:
        if what == "record":
            home = a if home is None else home
            records[b] = a
        elif what in ("launch", "graph"):
            worked[a] = True
            joined.discard(a)
        elif what == "wait" and a == home and b in records and records[b] != home:
            joined.add(records[b])
    worked.pop(home, None)
    return set(worked), joined


@pytest.mark.parametrize("what,n,graph", [("instantiate", 1, True), ("instantiate", 3, True), ("begin capture", 1, True),
                                          ("end capture", 2, True), ("graph", 1, True), ("graph", 5, True),
                                          ("launch", 40, False), ("launch", 7, False)])
def test_a_failing_call_leaves_no_stream_unjoined(env, what, n, graph):
    gpu, fake = env
    pool = make_pool(gpu, SIDES if graph else SIDES * 4)
    assert pool.sweep_groups == (4, 4)
    fake.reset()
    fake.fail(what, n)
    try:
        pool.run(2, graph=graph)
        failed = False
    except gpu.SU2GPUError:
        failed = True
    assert fake.failed(what)
    ops = fake.ops()
    captured = {a for w, a, _ in ops if w == "begin capture"}
    worked, joined = forked_and_joined(ops)
    worked -= captured  # what was launched there was captured, not run
    assert worked and worked <= joined
    # only launches that fail fail the run: without a graph its group's passes
    # are launched one by one
    assert failed == (what in ("graph", "launch"))
    # the next run is a normal one
    fake.reset()
    pool.run(2, graph=graph)
    worked, joined = forked_and_joined([o for o in fake.ops()])
    assert len(worked - captured) == 4 and worked - captured <= joined
    pool.close()


def test_a_run_without_a_graph_launches_every_sweep(env):
    gpu, fake = env
    pool = make_pool(gpu)
    fake.reset()
    fake.fail("instantiate", 1)  # the second group's
    pool.run(3)
    ops = fake.ops()
    captured = {a for w, a, _ in ops if w == "begin capture"}
    passes = pool.launches_per_sweep() // 4
    replays, launches = {}, {}
    for w, a, _ in ops:
        if w == "graph":
            replays[a] = replays.get(a, 0) + 1
        if w == "launch" and a not in captured:
            launches[a] = launches.get(a, 0) + 1
    assert sorted(replays.values()) == [3, 3, 3] and list(launches.values()) == [3 * passes]
    pool.close()


def test_groups_off_is_off(env):
    gpu, fake = env
    pool = make_pool(gpu)
    assert pool.sweep_groups == (4, 4)  # the automatic choice
    for off in (None, (1, 3), (0, 1), (-1, 1)):
        pool.sweep_groups = (3, 2)
        assert pool.sweep_groups == (3, 2)
        pool.sweep_groups = off
        assert pool.sweep_groups == (0, 1)
        fake.reset()
        pool.run(2)
        assert len({a for w, a, _ in fake.ops() if w == "graph"}) == 1
    # off does not depend on the other mode, and stays until it is set again
    pool.persistent = False
    pool.persistent = None
    assert pool.sweep_groups == (0, 1)
    pool.sweep_groups = (2, 2)
    assert pool.sweep_groups == (2, 2)
    pool.close()


def test_autotuner_with_groups_fixed_off(env, monkeypatch):
    gpu, fake = env
    pool = make_pool(gpu, SIDES * 2)
    monkeypatch.setenv("SU2GPU_SWEEP_GROUPS", "1,1")
    pool.autotune()
    assert pool.sweep_groups == (0, 1)
    pool.close()


def test_autotuner_again_compares_with_the_automatic_choice(env):
    gpu, fake = env

    def captures(groups):
        pool = make_pool(gpu, SIDES * 2)
        if groups:
            pool.sweep_groups = groups
        fake.reset()
        pool.autotune()  # every launch takes the same time: nothing is picked
        n = sum(w == "begin capture" for w, _, _ in fake.ops())
        left = pool.sweep_groups
        pool.close()
        return n, left

    assert captures((5, 3)) == captures(None)


def test_failed_autotuner_leaves_the_groups(env):
    gpu, fake = env
    pool = make_pool(gpu, SIDES * 2)
    pool.sweep_groups = (5, 3)
    fake.reset()
    fake.fail("instantiate", 6)
    with pytest.raises(gpu.SU2GPUError):
        pool.autotune()
    assert fake.failed("instantiate") and pool.sweep_groups == (5, 3)
    pool.close()


def streams_launched_on(fake, pool, graph):
    fake.reset()
    pool.run(1, graph=graph)
    captured = {a for w, a, _ in fake.ops() if w == "begin capture"}
    return len({a for w, a, _ in fake.ops() if w == "graph" or (w == "launch" and a not in captured)})


@pytest.mark.parametrize("precision,copies,direct", [(32, 1, 1), (32, 3, 1), (32, 4, 4), (64, 1, 4)])
def test_direct_launches_of_small_pools_are_not_grouped(env, precision, copies, direct):
    # 0.1 M sites a copy; a pool's groups run side by side from 0.4 M on, FP64
    # ones always
    gpu, fake = env
    pool = make_pool(gpu, SIDES * copies, precision=precision)
    assert pool.sweep_groups == (4, 4)
    assert streams_launched_on(fake, pool, False) == direct
    pool.sweep_groups = (3, 2)  # what the caller asks for holds either way
    assert streams_launched_on(fake, pool, False) == 2
    pool.close()


@pytest.mark.parametrize("groups,turns", [(4, False), (10, True)])
def test_conversions_of_a_large_cycle_do_not_wait_behind_the_sweeps(env, monkeypatch, groups, turns):
    # the sweeps' passes always have blocks waiting for room: a transfer stream
    # of lower priority gets none until the sweeps of the groups in flight end
    gpu, fake = env
    monkeypatch.setenv("SU2GPU_CYCLE_GROUPS", str(groups))
    sides = [(4, 6, 8)] * 15
    pool = make_pool(gpu, sides)
    fields = [{"link": np.zeros((192, 3, 4)), "trip": np.zeros((192, 3))} for _ in sides]
    pool.cycle(list(pool.active()), fields, 2)
    priority = {a: b for w, a, b in fake.ops() if w == "stream"}
    swept = {a for w, a, _ in fake.ops() if w == "graph"}
    moved = {a for w, a, _ in fake.ops() if w == "copy"} & set(priority) - swept
    moved = {a for a in moved if sum(w == "copy" and x == a for w, x, _ in fake.ops()) >= len(sides)}
    assert swept and len(moved) == 2  # upload and download streams
    assert (max(priority[a] for a in moved) <= min(priority[a] for a in swept)) == turns  # less is higher
    pool.close()


@pytest.mark.parametrize("n", [0, 1, 2])
def test_a_failing_team_leaves_no_stream_unjoined(env, n):
    gpu, fake = env
    pool = make_pool(gpu, [(4, 4, 4), (8, 8, 8), (8, 8, 16)])
    assert pool.launches_per_sweep() == 3  # two shapes, and the sweep counters
    fake.reset()
    fake.fail("launch", n)
    with pytest.raises(gpu.SU2GPUError):
        pool.run(2)
    worked, joined = forked_and_joined(fake.ops())
    assert worked <= joined and len(joined) == 2
    fake.reset()
    pool.run(2)
    pool.close()


@pytest.mark.parametrize("what,n", [("copy", 3), ("copy", 20), ("copy", 31), ("launch", 2), ("launch", 9), ("graph", 5),
                                    ("wait", 12)])
def test_a_failing_cycle_returns_with_nothing_in_flight(env, monkeypatch, what, n):
    # its copies read and write the caller's arrays
    gpu, fake = env
    monkeypatch.setenv("SU2GPU_CYCLE_GROUPS", "4")
    sides = [(4, 6, 8)] * 8
    pool = make_pool(gpu, sides)
    fields = [{"link": np.zeros((192, 3, 4)), "trip": np.zeros((192, 3))} for _ in sides]
    pool.cycle(list(pool.active()), fields, 2)  # graphs, rings and tables are made
    fake.reset()
    fake.fail(what, n)
    with pytest.raises(gpu.SU2GPUError):
        pool.cycle(list(pool.active()), fields, 2)
    assert fake.failed(what)
    busy = set()
    for w, a, _ in fake.ops():
        if w in ("copy", "fill", "launch", "graph"):
            busy.add(a)
        if w == "sync":
            busy.discard(a)
    assert not busy
    pool.close()
