"""Rounding of the FP64 overrelaxation: the doublet's proposals with unit links
against long double, whose root mean square distance, in units of 2^-53 of a
proposal's length, is the update's own.  A form with the root and a division per
component, rounded each, measures 1.30; one that takes |s| as s^2 rsqrt(s^2)
1.45.  The line lies half-way; the mean is over 11520 sites, so it moves by less
than a hundredth from one configuration to another."""
import numpy as np
import pytest

from su2higgs_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.1, 0.4, 2.0])
def test_doublet_proposals_round_like_divisions(scale):
    from su2higgs_gb300 import gpu
    ld = np.longdouble
    err = []
    for seed in range(3):
        p = abi.make_params("fund", L=(16, 12, 20))
        lat = gpu.Lattice(p, seed=1)
        V = p.sites()
        nx, pv, _, _ = lat.layout_tables()
        link = np.zeros((V, 3, 4))
        link[..., 0] = 1.0
        phi = scale * np.random.default_rng(seed).normal(size=(V, 4))
        lat.upload(link=link, d0=phi)
        phi = phi.astype(ld)
        s = -sum(phi[nx[:, d]] + phi[pv[:, d]] for d in range(3))
        F = np.sqrt(np.sum(s * s, axis=1))
        e = s / F[:, None]
        X = np.sum(phi * e, axis=1)
        Y2 = np.sum((phi - X[:, None] * e) ** 2, axis=1)
        B, C = ld(0.5) * ld(p.msq_phi) + 3, ld(0.25) * ld(p.lambda_phi)
        cc = B + 2 * Y2 * C
        a, b, c, d = C, C * X, cc + C * X * X, F + cc * X + C * X ** 3
        x = -d / c
        for _ in range(60):
            x = x - (((a * x + b) * x + c) * x + d) / ((3 * a * x + 2 * b) * x + c)
        want = -phi + (X + x)[:, None] * e
        got = lat.site_values("or_doublet")
        err.append(np.linalg.norm((got - want).astype(float), axis=1) / np.linalg.norm(want.astype(float), axis=1))
        lat.close()
    rms = np.sqrt(np.mean(np.concatenate(err) ** 2)) * 2.0 ** 53
    assert rms < 1.38, rms
