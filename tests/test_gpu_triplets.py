"""The fused triplet kernel (k_efs_tri) at the sizes and bases where it can go
wrong: neighbour counts around its lane, stripe and list edges (0 and 1
neighbour up to past its capacity of 128), 1 to 3 species, exponents that
need more squarings or fall back, 8 exponents, other zeta and other function
tables, and networks of odd and large width.  Energies, forces and virial
are held to the plain path's bar against the oracle (1e-10 relative energy,
1e-9 eV/A), the two kernel families to each other at 100 times the rounding
of a sum of a few thousand terms."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu

SPC = [29, 46, 47]


def _check(tmp_path, monkeypatch, w, ns, basis, h=(10, 10), seed=3):
    import maise_b200
    from maise_b200 import models

    ND = int(w["ND"])
    path = str(tmp_path / "model")
    models.random_model(path, SPC[:ns], basis, (w["X"], w["LAT"], w["atmn"], max(ND, 1)), h=h, seed=seed)
    want = Oracle(path).efs(w["X"], w["LAT"], w["atmn"], ND, NM=400)
    args = (w["X"], w["LAT"], w["atmn"])
    out = []
    for legs, shape in (("1", "0"), ("1", "2"), ("1", "3"), ("1", "4"), ("0", "2")):
        monkeypatch.setenv("MAISE_B200_LEGS", legs)
        monkeypatch.setenv("MAISE_B200_SHAPE", shape)
        with maise_b200.Potential(path) as pot:
            r = pot.efs(*args, ND=ND, NM=400)
            G = pot.descriptors(*args, ND=ND, NM=400)
            out.append((r, G))
        what = f"legs {legs} shape {shape}"
        assert r["H"] == pytest.approx(want["H"], rel=1e-10), what
        np.testing.assert_allclose(r["F"], want["F"], atol=1e-9, err_msg=what)
        np.testing.assert_allclose(r["U"], want["U"], rtol=1e-10, atol=1e-9, err_msg=what)
    plain = out[-1]
    for r, G in out[:-1]:
        np.testing.assert_allclose(G, plain[1], rtol=1e-12, atol=1e-13 * max(1.0, np.abs(plain[1]).max()))
        np.testing.assert_allclose(r["F"], plain[0]["F"], atol=1e-11 * max(1.0, np.abs(plain[0]["F"]).max()))


def _cluster(n, ns, seed, spread):
    """n atoms on a jittered grid around the first, so that it has n - 1 neighbours."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.array([[i, j, k] for i in range(m) for j in range(m) for k in range(m)], float) - (m - 1) / 2
    g = g[np.argsort((g ** 2).sum(1), kind="stable")[:n]] * spread
    X = g + rng.normal(0, 0.05, (n, 3)) + 20.0
    spc = np.sort(rng.integers(0, ns, n)).astype(np.int32)
    return dict(X=X, LAT=np.eye(3) * 40.0, atmn=spc, ND=0)


@pytest.mark.parametrize("ns", [1, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 9, 32, 33, 34, 65, 66, 97, 128, 129, 130, 140])
def test_neighbour_counts(tmp_path, monkeypatch, n, ns):
    """Descriptors and their VJP (no network in between) in clusters where
    every atom neighbours every other one."""
    import maise_b200
    from maise_b200 import models, workloads

    w = _cluster(n, ns, 10 * n + ns, 1.6 if n < 60 else 1.25)
    ref = workloads.random_alloy(n=2, a=3.7, seed=6, species=SPC[:ns], jitter=0.1)
    path = str(tmp_path / "model")
    models.random_model(path, SPC[:ns], models.Basis(), (ref["X"], ref["LAT"], ref["atmn"], 3), seed=3)
    o = Oracle(path)
    args = (w["X"], w["LAT"], w["atmn"])
    G = np.asarray(o.descriptors(*args, 0, NM=400)).reshape(n, -1)
    g = np.random.default_rng(n).normal(size=G.shape)
    F, U = o.vjp(*args, 0, g, NM=400)
    F, U = np.asarray(F).reshape(n, 3), np.asarray(U)
    # at most 8000 triplets of 43 terms an atom: a relative 1e-12 of the largest, with a margin of 10
    tol = 1e-11 * max(np.abs(U).max(), np.abs(F).max(), 1e-3)
    for legs, shape in (("1", "0"), ("1", "2"), ("1", "3"), ("1", "4"), ("0", "2")):
        monkeypatch.setenv("MAISE_B200_LEGS", legs)
        monkeypatch.setenv("MAISE_B200_SHAPE", shape)
        with maise_b200.Potential(path) as pot:
            np.testing.assert_allclose(pot.descriptors(*args, ND=0, NM=400), G, rtol=1e-11,
                                       atol=1e-13 * max(1.0, np.abs(G).max()))
            f, u = pot.descriptor_vjp(*args, g, ND=0, NM=400)
        np.testing.assert_allclose(f, F, atol=tol, err_msg=f"legs {legs} shape {shape}")
        np.testing.assert_allclose(u, U, atol=tol, err_msg=f"legs {legs} shape {shape}")


@pytest.mark.parametrize("kw", [
    dict(eta4=np.geomspace(0.004, 0.06, 7)),                          # 3 squarings
    dict(eta4=np.geomspace(0.004, 0.12, 7)),                          # 4 squarings
    dict(eta4=np.geomspace(0.004, 0.25, 7)),                          # beyond the polynomial: general kernel
    dict(eta4=np.geomspace(0.03, 0.003, 7)),                          # descending exponents
    dict(eta4=np.geomspace(0.003, 0.03, 8), g4_rows=[(e, z, l) for e in range(8) for z in range(4) for l in range(2)]),
    dict(eta4=[0.01], g4_rows=[(0, z, l) for z in range(4) for l in range(2)]),
    dict(zetas=(1.0, 3.0, 5.0, 8.0)),
    dict(zetas=(2.0,), lambdas=(1.0,), g4_rows=[(e, 0, 0) for e in range(7)]),
    dict(g4_rows=[(e, z, l) for e in range(7) for z in range(4) for l in range(2)] + [(2, 1, 0)]),  # a function twice
    dict(rc=4.5, eta2=np.geomspace(0.01, 0.9, 10)),
], ids=lambda kw: "-".join(f"{k}{len(v) if hasattr(v, '__len__') else v}" for k, v in kw.items()))
def test_bases(tmp_path, monkeypatch, kw):
    from maise_b200 import models, workloads

    w = workloads.random_alloy(n=2, a=3.7, seed=6, jitter=0.1)
    _check(tmp_path, monkeypatch, w, 3, models.Basis(**kw))


@pytest.mark.parametrize("h", [(1, 1), (7, 5), (16, 16), (17, 32), (32, 9)])
def test_network_widths(tmp_path, monkeypatch, h):
    from maise_b200 import models, workloads

    w = workloads.random_alloy(n=2, a=3.9, seed=8, species=(29, 46), jitter=0.1)
    _check(tmp_path, monkeypatch, w, 2, models.Basis(), h=h)


@pytest.mark.parametrize("a", [3.61, 3.3, 3.1, 2.9])
def test_dense_crystals(tmp_path, monkeypatch, a):
    """About 80 to 150 neighbours, the last past the kernel's capacity."""
    from maise_b200 import models, workloads

    w = workloads.fcc_supercell(n=2, a=a, jitter=0.05, seed=2)
    _check(tmp_path, monkeypatch, w, 1, models.Basis())
