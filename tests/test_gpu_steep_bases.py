"""Bases whose G4 exponents are too steep for the fused kernel's polynomial
(or negative) run on that kernel too, with exp() in the polynomial's place.
The bars are the plain path's against the oracle: 1e-10 relative energy,
1e-9 eV/A and descriptors to 1e-11 of their sums of a few thousand terms."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu

ALL8 = [(e, z, l) for e in range(8) for z in range(4) for l in range(2)]


@pytest.mark.parametrize("ns", [1, 3])
@pytest.mark.parametrize("kw", [
    dict(eta4=np.geomspace(0.004, 0.0312, 7)),               # just past the polynomial's range
    dict(eta4=np.geomspace(0.004, 0.126, 7)),
    dict(eta4=np.geomspace(0.01, 1.0, 7)),
    dict(eta4=[40.0], g4_rows=[(0, z, l) for z in range(4) for l in range(2)]),  # factors that underflow
    dict(eta4=np.geomspace(0.01, 1.0, 8), g4_rows=ALL8),     # another function table: the general form
    dict(eta4=np.geomspace(0.01, 1.0, 7), zetas=(1.0, 3.0, 5.0, 8.0)),
    dict(eta4=[-0.002, 0.0, 0.01, 0.02, 0.03, 0.04, 0.05]),
], ids=["edge", "past", "steep", "underflow", "eight", "zetas", "negative"])
def test_steep_bases(tmp_path, monkeypatch, kw, ns):
    import maise_b200
    from maise_b200 import models, workloads

    spc = [29, 46, 47][:ns]
    w = workloads.random_alloy(n=2, a=3.7, seed=6, species=tuple(spc), jitter=0.1)
    args = (w["X"], w["LAT"], w["atmn"])
    path = str(tmp_path / "model")
    models.random_model(path, spc, models.Basis(**kw), args + (3,), seed=3)
    o = Oracle(path)
    want = o.efs(*args, 3, NM=400)
    G = np.asarray(o.descriptors(*args, 3, NM=400)).reshape(len(w["atmn"]), -1)
    assert np.isfinite(want["H"]) or (min(kw["eta4"]) < 0 and ns > 1)
    for shape in ("0", "2", "3", "4"):
        monkeypatch.setenv("MAISE_B200_SHAPE", shape)
        with maise_b200.Potential(path) as pot:
            r = pot.efs(*args, NM=400)
            np.testing.assert_allclose(pot.descriptors(*args, NM=400), G, rtol=1e-11,
                                       atol=1e-13 * max(1.0, np.abs(G).max()))
            # a negative exponent's mixed-species exponent is not a number, which the
            # general kernel keeps as the reference does
            assert all(e["legs"] == np.isfinite(want["H"]) for e in pot.tune_table())
        np.testing.assert_allclose(r["H"], want["H"], rtol=1e-10, err_msg=shape)
        np.testing.assert_allclose(r["F"], want["F"], atol=1e-9, err_msg=shape)
        np.testing.assert_allclose(r["U"], want["U"], rtol=1e-10, atol=1e-9, err_msg=shape)


def _exact_g4(basis, X, rc, eta):
    """G4 of every atom of a one-species cluster in long double, [N, ng4]."""
    LD = np.longdouble
    X = X.astype(LD)
    pi = LD(np.pi) + LD(1.2246467991473532e-16)

    def fc(r):
        return LD(0.5) * (1 + np.cos(pi * r / LD(rc)))

    out = np.zeros((len(X), basis.ng4), LD)
    for i in range(len(X)):
        d = np.delete(X, i, 0) - X[i]
        r = np.sqrt((d * d).sum(1))
        d, r = d[r < rc], r[r < rc]
        a, b = np.triu_indices(len(r), 1)
        s = np.sqrt(((d[a] - d[b]) ** 2).sum(1))
        a, b, s = a[s < rc], b[s < rc], s[s < rc]
        c = (d[a] * d[b]).sum(1) / (r[a] * r[b])
        A, rho = 2 * fc(r[a]) * fc(r[b]) * fc(s), r[a] ** 2 + r[b] ** 2 + s ** 2
        for f, (e, z, l) in enumerate(basis.g4):
            zeta = LD(basis.zetas[z])
            out[i, f] = (A * np.exp(-LD(eta[e]) * rho) * LD(2) ** (1 - zeta) * (1 + LD(basis.lambdas[l]) * c) ** zeta).sum()
    return out


@pytest.mark.parametrize("top", [0.05, 0.12, 1.0])
def test_precision_of_steep_descriptors(tmp_path, top):
    """Against long double: the stored descriptor's own rounding and one more,
    1.1e-16 each, in the norm over atoms and functions.  (A polynomial squared
    three or four times had 3.4e-16 and 7.4e-16.)"""
    import maise_b200
    from maise_b200 import models

    g = np.array([[i, j, k] for i in range(4) for j in range(4) for k in range(4)], float) * 2.3
    X = g + np.random.default_rng(3).normal(0, 0.1, g.shape) + 20.0
    basis = models.Basis(eta4=np.geomspace(0.004, top, 7))
    args = (X, np.eye(3) * 60.0, np.zeros(len(X), np.int32))
    path = str(tmp_path / "model")
    models.random_model(path, [29], basis, args + (1,), seed=3)
    bohr = float(f"{models.BOHR:.9f}")  # the file's digits
    eta = [float(f"{v * models.BOHR ** 2:.12f}") / (bohr * bohr) for v in basis.eta4]
    want = _exact_g4(basis, X, float(f"{basis.rc / models.BOHR:.12f}") * bohr, eta)
    with maise_b200.Potential(path) as pot:
        got = pot.descriptors(*args, ND=0)[:, basis.ng2:]
    assert float(np.linalg.norm((got - want).astype(float)) / np.linalg.norm(want.astype(float))) < 2.2e-16
