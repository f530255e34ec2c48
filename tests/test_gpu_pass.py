"""The ends of a single-structure pass: the all-pairs neighbour list at the
image counts where its two walks switch, in the reference's order (atom, then
image) and set, against plain numpy; and the totals, which several CTAs sum,
against the per-atom energies and the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _list(X, L, ND, rc):
    """Per atom (j, image) in order of j, then images, as LIST walks them."""
    R = np.linalg.inv(L).T
    nq = [int(np.ceil(rc * np.linalg.norm(R[q]))) if q < ND else 0 for q in range(3)]
    img = np.array([[a, b, c] for a in range(-nq[0], nq[0] + 1) for b in range(-nq[1], nq[1] + 1)
                    for c in range(-nq[2], nq[2] + 1)])
    out = []
    for i in range(len(X)):
        rows = []
        for j in range(len(X)):
            d = (img @ L) + (X[j] - X[i])
            ok = (d * d).sum(1) < rc * rc
            if i == j:
                ok &= (img != 0).any(1)
            rows += [(j, *s) for s in img[ok]]
        out.append(rows)
    return out, len(img)


@pytest.mark.parametrize("cell,ND,n", [
    ((30.0, 30.0, 30.0), 0, 7),     # a cluster: no images
    ((7.0, 30.0, 30.0), 1, 5),      # 3
    ((7.0, 7.5, 30.0), 2, 6),       # 9
    ((4.0, 7.5, 30.0), 2, 6),       # 15
    ((7.0, 7.5, 8.0), 3, 9),        # 27: the images fit a warp
    ((4.0, 7.5, 8.0), 3, 6),        # 45
    ((4.0, 4.2, 4.5), 3, 4),        # 125
    ((2.9, 4.2, 4.5), 3, 3),        # 175: more than the lanes hold
    ((2.7, 2.8, 2.9), 3, 1),        # 343
])
def test_all_pairs_list(tmp_path, cell, ND, n):
    import maise_b200
    from maise_b200 import models, workloads

    w = workloads.random_alloy(n=2, a=3.8, seed=1, species=(29, 46), jitter=0.05)
    path = models.random_model(str(tmp_path / "model"), [29, 46], models.Basis(), (w["X"], w["LAT"], w["atmn"], 3))
    rng = np.random.default_rng(n)
    L = np.diag(cell) + np.array([[0, 0, 0], [0.2, 0, 0], [0.1, -0.3, 0]])
    X = rng.uniform(0.01, 0.99, (n, 3)) @ L
    if ND == 0:
        X = 15.0 + rng.uniform(-4, 4, (n, 3))
    with maise_b200.Potential(path) as pot:
        nn, nj, sh, Xw = pot.neighbours(X, L, np.zeros(n, np.int32), ND=ND, NM=900, path=1)
        want, nimg = _list(Xw, L, ND, pot.rc)
    assert nimg == {(30.0, 30.0, 30.0): 1, (7.0, 30.0, 30.0): 3, (7.0, 7.5, 30.0): 9}.get(cell, nimg)
    for i in range(n):
        got = [(int(nj[i, t]), *map(int, sh[i, t])) for t in range(nn[i])]
        assert got == [tuple(map(int, r)) for r in want[i]], (cell, i)


@pytest.mark.parametrize("N", [1, 31, 255, 257, 512, 513, 1025])
def test_totals(tmp_path, monkeypatch, N):
    import maise_b200
    from maise_b200 import models, workloads

    w = workloads.fcc_particle(n_target=2400, seed=4, species=(29, 46))
    X = w["X"][np.argsort(np.linalg.norm(w["X"] - w["X"].mean(0), axis=1), kind="stable")[:N]]
    spc = np.sort(np.arange(N) % 2).astype(np.int32)
    ref = workloads.random_alloy(n=2, a=3.9, seed=1, species=(29, 46), jitter=0.1)
    path = models.random_model(str(tmp_path / "model"), [29, 46], models.Basis(),
                               (ref["X"], ref["LAT"], ref["atmn"], 3))
    # one shape for both modes: the autotuner may choose different ones, whose sums round differently
    monkeypatch.setenv("MAISE_B200_SHAPE", "3")
    with maise_b200.Potential(path) as pot:
        first = pot.efs(X, w["LAT"], spc, ND=0, NM=200)
        for _ in range(3):  # plain launches, capture, replay
            r = pot.efs(X, w["LAT"], spc, ND=0, NM=200)
            e = pot.energy(X, w["LAT"], spc, ND=0, NM=200)
            np.testing.assert_array_equal(r["X"], X)
            np.testing.assert_array_equal(r["EA"], first["EA"])
            np.testing.assert_array_equal(e["EA"], first["EA"])
            assert r["E"] == pytest.approx(first["EA"].sum(), rel=1e-13)
            assert e["E"] == r["E"]
            scale = max(1.0, np.abs(first["F"]).max())
            np.testing.assert_allclose(r["F"], first["F"], atol=1e-12 * scale)
            np.testing.assert_allclose(r["F"].sum(0), 0.0, atol=1e-11 * scale * N)
            np.testing.assert_allclose(r["U"], first["U"], rtol=1e-11, atol=1e-10)
