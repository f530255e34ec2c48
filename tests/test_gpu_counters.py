"""The pair and triplet counters of mb_profile: every pass that lists an atom's
triplets counts them, the VJP's as well as the forward ones, on the fused kernel
at any of its shapes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["0", "1", "2", "3", "4"])
def test_every_mode_counts_its_triplets(tmp_path, monkeypatch, shape):
    import maise_b200
    from maise_b200 import models, workloads

    w = workloads.random_alloy(n=2, a=3.7, seed=6, jitter=0.1)
    args = (w["X"], w["LAT"], w["atmn"])
    path = str(tmp_path / "model")
    models.random_model(path, [29, 46, 47], models.Basis(), args + (3,), seed=3)
    monkeypatch.setenv("MAISE_B200_SHAPE", shape)
    with maise_b200.Potential(path) as pot:
        nn, nj, sh, X = pot.neighbours(*args)
        # triplets: pairs of an atom's neighbours within the cutoff of each other
        rc, want = 6.0, 0
        for i in range(len(X)):
            d = X[nj[i, :nn[i]]] + sh[i, :nn[i]] @ np.asarray(w["LAT"]) - X[i]
            r = np.linalg.norm(d[:, None] - d[None], axis=-1)
            want += int((r[np.triu_indices(len(d), 1)] < rc).sum())
        pot.efs(*args)  # the neighbour capacity is settled
        g = np.ones((len(X), pot.D))
        for call in (lambda: pot.efs(*args), lambda: pot.energy(*args), lambda: pot.descriptors(*args),
                     lambda: pot.descriptor_vjp(*args, g)):
            pot.profile(True)
            call()
            c = pot.profile_read()
            assert (c["launches"], c["pairs"], c["triplets"]) == (1, int(nn.sum()), want)
