"""The autotuner's table: one handle taken through more (mode, size bucket,
neighbour capacity) keys than any table holds still computes what a fresh
handle and the oracle do.  The trial launches of a key that finds the table
full must not add to the forces."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu

CAPACITIES = (72, 80, 88, 96)
SIZES = (1, 2, 4, 8, 16, 32, 64, 128, 256)  # a bucket each; 4 modes: 144 keys in all


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    from maise_b200 import models, workloads

    w = workloads.random_alloy(n=2, a=3.7, seed=6, jitter=0.1)
    path = str(tmp_path_factory.mktemp("tuner") / "model")
    models.random_model(path, [29, 46, 47], models.Basis(), (w["X"], w["LAT"], w["atmn"], 3), seed=3)
    return path, w


@pytest.fixture
def worn(model):
    """A handle that has met 144 keys, at a capacity it has no key for."""
    import maise_b200

    pot = maise_b200.Potential(model[0])
    for cap in CAPACITIES:
        pot.reserve(256, cap)
        for n in SIZES:
            rng = np.random.default_rng(n)
            X = rng.uniform(0, 2, (n, 3)) + 3.0 * np.arange(n)[:, None] * [1.0, 0.0, 0.0]
            args = (X, np.eye(3) * 900.0, np.zeros(n, np.int32))
            pot.efs(*args, ND=0)
            pot.energy(*args, ND=0)
            pot.descriptors(*args, ND=0)
            pot.descriptor_vjp(*args, rng.normal(size=(n, pot.D)), ND=0)
    pot.reserve(256, 104)
    yield pot
    pot.close()


def test_forces_after_many_keys(model, worn):
    import maise_b200

    path, w = model
    args = (w["X"], w["LAT"], w["atmn"])
    o = Oracle(path)
    want = o.efs(*args, 3, NM=400)
    g = np.random.default_rng(1).normal(size=(len(w["atmn"]), worn.D))
    wantF, wantU = o.vjp(*args, 3, g, NM=400)
    v = np.random.default_rng(2).normal(0, 1e-3, w["X"].shape)
    got = worn.efs(*args, ND=3)
    F, U = worn.descriptor_vjp(*args, g, ND=3)
    md = worn.md_nvt(*args, v, 300.0, nsteps=7)
    with maise_b200.Potential(path) as fresh:
        wmd = fresh.md_nvt(*args, v, 300.0, nsteps=7)
    assert got["H"] == pytest.approx(want["H"], rel=1e-10)
    np.testing.assert_allclose(got["F"], want["F"], atol=1e-9)
    np.testing.assert_allclose(got["U"], want["U"], rtol=1e-10, atol=1e-9)
    tol = 1e-11 * max(np.abs(wantF).max(), np.abs(wantU).max())
    np.testing.assert_allclose(F, np.asarray(wantF).reshape(-1, 3), atol=tol)
    np.testing.assert_allclose(U, wantU, atol=tol)
    # seven steps of 1 fs: forces that agree to 1e-9 eV/A move an atom by less than 1e-12 A
    np.testing.assert_allclose(md["X"], wmd["X"], atol=1e-10)


def test_new_key_is_recorded(model, worn):
    """A key met after the table is full is kept, so its shapes are not timed
    again on the next call (which then runs as a graph)."""
    _, w = model
    args = (w["X"], w["LAT"], w["atmn"])
    for mode, call in (("efs", worn.efs), ("energy", worn.energy), ("descriptors", worn.descriptors)):
        call(*args, ND=3)
        assert [e for e in worn.tune_table() if (e["mode"], e["size_bucket"], e["capacity"]) == (mode, 5, 104)], mode
