"""The surrogate's histogram where the lanes a pair of atoms takes change: cells
with 1, 3, 5, 7, 9 and 19 or more images in reach (rmax 6 A), atom counts that
leave the last step ragged, and the largest count; at test_gpu_screen.py's
tolerances against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import surrogate as su

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell", [(60.0, 60.0, 60.0), (3.0, 60.0, 60.0), (25.0, 25.0, 25.0), (16.0, 16.0, 16.0),
                                  (9.0, 9.0, 60.0), (9.0, 9.0, 13.0), (10.0, 10.0, 10.0)])
@pytest.mark.parametrize("n,nspc", [(1, 1), (2, 3), (7, 4), (33, 2), (61, 3)])
def test_features_by_image_count(cell, n, nspc):
    from maise_b200.surrogate import Surrogate

    rng = np.random.default_rng(n)
    lat = np.diag(cell)
    X = rng.uniform(0, 1, (n, 3)) @ np.diag(np.minimum(cell, 14.0))
    s = dict(X=X, LAT=lat, atmn=np.sort(rng.integers(0, nspc, n)).astype(np.int32))
    sur = Surrogate(nspc)
    got = sur.features([s, s])
    sur.close()
    want = su.rdf_features(s["X"], lat, s["atmn"], nspc)
    for g in got:
        np.testing.assert_allclose(g, want, rtol=1e-5, atol=1e-6 * max(1.0, np.abs(want).max()))


def test_features_of_the_largest_structure():
    from maise_b200.surrogate import Surrogate

    rng = np.random.default_rng(5)
    n, b = 256, 15.7
    s = dict(X=rng.uniform(0, b, (n, 3)), LAT=b * np.eye(3), atmn=np.sort(rng.integers(0, 3, n)).astype(np.int32))
    sur = Surrogate(3)
    got = sur.features([s])[0]
    sur.close()
    want = su.rdf_features(s["X"], s["LAT"], s["atmn"], 3)
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-6 * max(1.0, np.abs(want).max()))
