"""The one-CTA cell build at its edges: one atom, fewer and more atoms than
threads, its largest size and one past it, atoms all in one bin.  The lists
through the cells hold exactly the all-pairs lists' entries."""
from __future__ import annotations

import neighbour_cases as nc
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pot(tmp_path_factory):
    import maise_b200
    from maise_b200 import models, workloads

    d = tmp_path_factory.mktemp("cell_model")
    w = workloads.fcc_supercell(n=2, a=3.61, jitter=0.05, seed=0)
    models.random_model(str(d / "model"), [29], models.Basis(), (w["X"], w["LAT"], w["atmn"], 3), seed=1)
    with maise_b200.Potential(str(d / "model")) as p:
        yield p


@pytest.mark.parametrize("spacing,n", [(3.3, 1), (3.3, 31), (3.3, 1023), (3.3, 1025), (3.3, 4096), (3.3, 4097),
                                       (1.2, 64)])
def test_cell_build(pot, spacing, n):
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1 / 3)))
    X = np.array([[i, j, k] for i in range(m) for j in range(m) for k in range(m)], float) * spacing
    X = X[rng.permutation(len(X))[:n]] + rng.normal(0, 0.1, (n, 3)) + 0.5
    L = np.eye(3) * max(19.0, m * 3.3 + 0.1)
    got = [pot.neighbours(X, L, np.zeros(n, np.int32), ND=3, NM=100, path=p) for p in (1, 2)]
    want, cells = (nc.multiset(*g[:3]) for g in got)
    assert want == cells
    again = pot.neighbours(X, L, np.zeros(n, np.int32), ND=3, NM=100, path=2)
    for a, b in zip(got[1], again):
        assert np.array_equal(a, b)  # the order too repeats
