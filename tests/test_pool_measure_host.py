"""Where the pool's measurement writes its sums, on a CUDA runtime that runs
nothing (fake_gpu.py): into the sums' buffer as it is after the pool's tables have
been made for its present chains -- on a pool that has never swept, and after
chains have been added."""
import pytest

from fake_gpu import fake_gpu
from su2higgs_gb300 import abi


@pytest.fixture
def env(monkeypatch, tmp_path_factory):
    return fake_gpu(monkeypatch, tmp_path_factory.getbasetemp())


@pytest.mark.parametrize("precision", [32, 64])
def test_sums_go_to_the_present_buffer(env, precision):
    gpu, fake = env
    p = abi.make_params("adj", L=(4, 6, 8), precision=precision)
    pool = gpu.Pool(p, arena_bytes=16 * gpu.Pool.chain_bytes(p), max_chains=16)
    fake.watch("k_pool_reduce", 4)
    n = 0
    for more in (1, 2, 5, 8):
        for _ in range(more):
            pool.add(p, seed=n, chain=n)
            n += 1
        pool.measure()
        assert fake.room() >= n * abi.NMEAS * 8
    pool.close()
