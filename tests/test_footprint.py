"""su2gpu_footprint_bytes against what a context allocates, on a CUDA runtime that
runs nothing (fake_gpu.py)."""
import ctypes

import pytest

from fake_gpu import fake_gpu
from su2higgs_gb300 import abi


@pytest.fixture
def env(monkeypatch, tmp_path_factory):
    return fake_gpu(monkeypatch, tmp_path_factory.getbasetemp())


# around the sizes where the measurement's launch shape changes (38912 and 77824 sites)
@pytest.mark.parametrize("L", [(2, 2, 2), (8, 8, 8), (16, 16, 16), (32, 32, 38), (38, 32, 34), (64, 32, 38), (48, 48, 48)])
@pytest.mark.parametrize("content,precision", [("fund", 32), ("fund", 64), ("adj", 32), ("su2u1s", 64), ("higgs2", 32)])
def test_footprint_covers_what_a_lattice_holds(env, content, precision, L):
    gpu, fake = env
    p = abi.make_params(content, L=L, precision=precision)
    before = fake.live_bytes()
    lat = gpu.Lattice(p, seed=1)
    lat.run_sweeps(0, 1)
    lat.measure()
    held = fake.live_bytes() - before - p.sites() * 12 * 8  # without the upload's staging memory
    lat.close()
    said = gpu.lib().su2gpu_footprint_bytes(ctypes.byref(p))
    # every buffer is counted, the fields and a few pages apart no more than that
    assert held <= said <= held + 16384
    assert fake.live_bytes() == before
