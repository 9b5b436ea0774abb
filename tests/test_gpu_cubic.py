"""The FP64 overrelaxation root (polysolve3): Newton's method from the FP32
root, Cardano's formula in FP64 where that start is no good.  The triplet's
proposals with unit links against the root found in long double, from fields of
ordinary size (the usual start) to fields and couplings whose cubic overflows or
cancels in FP32.  The root is well conditioned (B > 0, C > 0: the cubic is
monotonic), so a proposal is within a few FP64 roundings of the exact one: 1e-13
of its length."""
import numpy as np
import pytest

from su2higgs_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,b4", [(0.4, 0.005), (0.4, 1e-14), (3.0, 2.0), (1e9, 1e-3), (1e18, 0.1), (1e-12, 0.1)])
def test_triplet_proposals(scale, b4):
    from su2higgs_gb300 import gpu
    L = (4, 6, 4)
    p = abi.make_params("adj", L=L, msq_triplet=-0.2, b4=b4)
    lat = gpu.Lattice(p, seed=1)
    V = p.sites()
    nx, pv, _, _ = lat.layout_tables()
    link = np.zeros((V, 3, 4))
    link[..., 0] = 1.0
    t = scale * np.random.default_rng(5).normal(size=(V, 3))
    lat.upload(link=link, trip=t)
    ld = np.longdouble
    t = t.astype(ld)
    s = -sum(t[nx[:, d]] + t[pv[:, d]] for d in range(3))
    F = np.sqrt(np.sum(s * s, axis=1))
    e = s / F[:, None]
    X = np.sum(t * e, axis=1)
    Y2 = np.sum((t - X[:, None] * e) ** 2, axis=1)
    B, C = ld(0.5) * ld(p.msq_triplet) + 3, ld(0.25) * ld(b4)
    cc = B + 2 * Y2 * C
    a, b, c, d = C, C * X, cc + C * X * X, F + cc * X + C * X ** 3
    x = -d / c
    for _ in range(300):
        x = x - (((a * x + b) * x + c) * x + d) / ((3 * a * x + 2 * b) * x + c)
    want = -t + (X + x)[:, None] * e
    got = lat.site_values("or_triplet")
    err = np.linalg.norm((got - want).astype(np.float64), axis=1) / np.linalg.norm(want.astype(np.float64), axis=1)
    assert np.all(np.isfinite(got)) and err.max() < 1e-13, err.max()
