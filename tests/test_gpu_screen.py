"""The surrogate's histogram and GEMM kernels where their rules switch,
against the oracle (oracle/surrogate.py), at that file's tolerances: cells
with more images in reach than the kernel lists, thin and skewed cells, one
atom, Gaussians narrower than a bin and wider than a group of lanes, four
species; layers wide enough for the 64 x 64 tiles and ragged ones below."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import surrogate as su

pytestmark = pytest.mark.gpu

CUBE = np.eye(3)
SKEW = np.array([[1.0, 0, 0], [0.48, 0.88, 0], [0.45, 0.3, 0.84]])


@pytest.mark.parametrize("lat,n", [(1.12 * CUBE, 1), (1.6 * SKEW, 1), (2.9 * SKEW, 3), (8.0 * SKEW, 20),
                                   (np.diag([1.5, 9.0, 14.0]), 5), (20.0 * CUBE, 12)])
@pytest.mark.parametrize("nspc,nbins,sigma", [(1, 128, 0.05), (2, 16, 0.05), (3, 128, 0.4), (4, 40, 0.3)])
def test_features_match_oracle(lat, n, nspc, nbins, sigma):
    from maise_b200.surrogate import Surrogate

    rng = np.random.default_rng(n + nbins)
    s = dict(X=rng.uniform(0, 1, (n, 3)) @ lat, LAT=lat, atmn=np.sort(rng.integers(0, nspc, n)).astype(np.int32))
    sur = Surrogate(nspc, nbins=nbins, sigma=sigma)
    got = sur.features([s])[0]
    sur.close()
    want = su.rdf_features(s["X"], s["LAT"], s["atmn"], nspc, nbins=nbins, sigma=sigma)
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-6 * max(1.0, np.abs(want).max()))


@pytest.mark.parametrize("B,hidden", [(1, (33, 31, 1)), (65, (64, 32, 16)), (1700, (400, 37, 8))])
def test_gradient_matches_oracle(B, hidden):
    from maise_b200.surrogate import Surrogate

    sur = Surrogate(2, nbins=37, hidden=hidden, seed=3)
    rng = np.random.default_rng(B)
    x = rng.normal(size=(B, sur.nin)).astype(np.float32)
    t = rng.normal(size=B).astype(np.float32)
    loss, g = sur.loss_grad(x, t)
    want_loss, want_g = su.mlp_loss_grad(sur.params.astype(np.float64), x.astype(np.float64), t.astype(np.float64),
                                         sur.nin, sur.hidden)
    sur.close()
    assert loss == pytest.approx(want_loss, rel=1e-5)
    np.testing.assert_allclose(g, want_g, atol=1e-4 * np.abs(want_g).max())
