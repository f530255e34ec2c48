"""RDFs and overlaps of EA members at the sizes where their kernels can go
wrong, against plain numpy in the same operation order: cells so thin that
the images outnumber the shared table of shifts, clusters, one atom, bins
and widths that give fewer and more than a warp of bins per pair; overlap
matrices around a tile's edges, split and unsplit sums, lengths of 1 up to
the reference's 9000 terms."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rdf(w, ns, nbins, rmin, rmax, sigma, ND):
    X, L, spc = np.asarray(w["X"]), np.asarray(w["LAT"]), np.asarray(w["atmn"])
    R = np.linalg.inv(L).T
    nq = [int(np.ceil(rmax * np.linalg.norm(R[q]))) if q < ND else 0 for q in range(3)]
    sh = np.array([[a, b, c] for a in range(-nq[0], nq[0] + 1) for b in range(-nq[1], nq[1] + 1)
                   for c in range(-nq[2], nq[2] + 1)], float) @ L
    npair = ns * (ns + 1) // 2
    out = np.zeros((npair, nbins))
    dr = rmax / nbins
    xk = np.arange(nbins) * dr
    with np.errstate(divide="ignore", invalid="ignore"):
        tap = np.where(xk < rmin, 1.0, np.cos(0.5 * np.pi * (xk - rmin) / (rmax - rmin)))
    Do = int(3.0 * sigma / dr)
    for i in range(len(X)):
        for j in range(len(X)):
            if spc[j] < spc[i]:
                continue
            r = np.linalg.norm(X[j] - X[i] + sh, axis=1)
            r = r[(r < rmax) & ((r > 1e-12) if i == j else True)]
            p = spc[i] * ns - spc[i] * (spc[i] - 1) // 2 + spc[j] - spc[i]
            for x in r:
                k = np.arange(max(0, int(x / dr) - Do), min(nbins - 1, int(x / dr) + Do) + 1)
                out[p, k] += tap[k] * np.exp(-(x - xk[k]) ** 2 * 0.5 / sigma ** 2) * (0.5 if spc[i] == spc[j] else 1.0)
    return out


@pytest.mark.parametrize("cell,ND,nbins,sigma", [
    ((9.0, 9.0, 9.0), 3, 3000, 0.008),
    ((2.1, 2.3, 2.2), 3, 3000, 0.008),   # 7 x 7 x 7 images: more than the shared table holds
    ((2.2, 9.0, 14.0), 3, 600, 0.008),   # fewer than a bin within 3 sigma
    ((12.0, 12.0, 12.0), 0, 3000, 0.05),  # a cluster; 151 bins a pair
    ((7.0, 8.0, 9.0), 2, 128, 0.05),
])
@pytest.mark.parametrize("n,ns", [(1, 1), (5, 2), (17, 3)])
def test_rdf_equals_numpy(cell, ND, nbins, sigma, n, ns):
    from maise_b200 import evos

    rng = np.random.default_rng(n + nbins)
    L = np.diag(cell) + np.array([[0, 0, 0], [0.3, 0, 0], [-0.2, 0.4, 0]])
    pop = [dict(X=rng.uniform(0, 1, (n, 3)) @ L, LAT=L, atmn=np.sort(rng.integers(0, ns, n)).astype(np.int32))
           for _ in range(2)]
    got = evos.rdf(pop, ns, nbins=nbins, sigma=sigma, normalise=False, ND=ND)
    for k, w in enumerate(pop):
        want = _rdf(w, ns, nbins, 5.8, 6.0, sigma, ND)
        # sums of a few hundred positive terms of rounding 1e-16 and an exponential of 1e-15 relative
        np.testing.assert_allclose(got[k], want, rtol=1e-11, atol=1e-12 * max(1.0, want.max()))


@pytest.mark.parametrize("S", [1, 7, 63, 64, 65, 130])
@pytest.mark.parametrize("T", [1, 31, 64, 65, 2047, 9000])
def test_overlaps_equal_numpy(S, T):
    from maise_b200 import evos

    R = np.random.default_rng(S * T).normal(size=(S, T))
    C = evos.overlaps(R)
    np.testing.assert_array_equal(C, C.T)
    np.testing.assert_allclose(C, R @ R.T, rtol=0, atol=1e-14 * T)


def test_overlaps_of_many_members():
    """Enough tiles that the sums are not split."""
    from maise_b200 import evos

    R = np.random.default_rng(3).normal(size=(1600, 96))
    np.testing.assert_allclose(evos.overlaps(R), R @ R.T, rtol=0, atol=1e-12)
