"""The batched FP32 evaluation where its triplet lists and tiles can go wrong:
0, 1 and a few neighbours, species blocks of odd sizes, a list longer than its
room (more than 2048 triplets of one atom), and bases on either side of the
rule that chooses the straight-line kernel.  Held to the FP64 one-structure
path at identical structures by the batched path's stated error (1e-5
eV/atom, 1e-4 eV/A), or, where forces are large, by 2e-5 of the largest: a
force is a sum of at most 3000 triplet terms of a few roundings of 6e-8 each,
which cancel to about a tenth of their size."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPC = [29, 46, 47]


def _blob(n, ns, spacing, box, seed):
    rng = np.random.default_rng(seed)
    g = np.array([[i, j, k] for i in range(4) for j in range(4) for k in range(4)], float)[:n]
    X = g * spacing + rng.normal(0, 0.03, (n, 3)) + 1.0
    return dict(X=X, LAT=np.diag(np.asarray(box, float)), atmn=np.sort(rng.integers(0, ns, n)).astype(np.int32))


def _check(tmp_path, structures, ns, basis):
    import maise_b200
    from maise_b200 import models

    big = max(structures, key=lambda s: len(s["atmn"]))
    path = str(tmp_path / "model")
    models.random_model(path, SPC[:ns], basis, (big["X"], big["LAT"], big["atmn"], 3), seed=9)
    with maise_b200.Potential(path) as pot:
        got = pot.efs_batch(structures)
        want = [pot.efs(s["X"], s["LAT"], s["atmn"], ND=3, NM=400) for s in structures]
    for k, (s, e) in enumerate(zip(structures, want)):
        n, top = len(s["atmn"]), max(np.abs(e["F"]).max(), 5.0)
        assert abs(got["H"][k] - e["H"]) / n <= 1e-5, k
        assert np.abs(got["F"][k] - e["F"]).max() <= 2e-5 * top, k
        assert np.abs(got["U"][k] - e["U"]).max() / n <= 2e-5 * max(np.abs(e["U"]).max() / n, 5.0), k


@pytest.mark.parametrize("ns", [1, 2, 3])
def test_neighbour_counts(tmp_path, ns):
    sizes = (1, 2, 3, 5, 8, 9, 17, 33, 47, 64)
    _check(tmp_path, [_blob(n, ns, 1.9, (30, 30, 30), n) for n in sizes], ns, _basis())


@pytest.mark.parametrize("ns", [1, 3])
def test_long_lists(tmp_path, ns):
    """About 90 neighbours on one side of an atom: 2700 triplets."""
    _check(tmp_path, [_blob(64, ns, 1.4, (30, 30, 8.0), 1), _blob(64, ns, 1.4, (30, 30, 8.5), 2)], ns, _basis())


@pytest.mark.parametrize("kw", [
    dict(eta4=np.geomspace(0.004, 0.06, 7)),                       # more squarings: the general kernel
    dict(eta4=[0.01, 0.02], g4_rows=[(0, 0, 0), (1, 1, 1)]),
    dict(eta4=[0.01], g4_rows=[(0, z, l) for z in range(4) for l in range(2)]),
    dict(g4_rows=[(e, z, l) for e in range(3, 7) for z in range(4) for l in range(2)] + [(4, 1, 0)]),
    dict(zetas=(1.0, 3.0, 5.0, 8.0)),
    dict(rc=4.5, eta2=np.geomspace(0.01, 0.9, 10)),
], ids=["eta-steep", "two-eta", "one-eta", "high-only", "zeta-odd", "rc-4.5"])
def test_bases(tmp_path, kw):
    from maise_b200 import models

    _check(tmp_path, [_blob(33, 2, 2.2, (9.2, 9.5, 9.9), 4)], 2, models.Basis(**kw))


def _basis():
    from maise_b200 import models

    return models.Basis()
