"""The batched FP32 evaluation has no systematic error beyond its rounding: over
a population the median error of the energy per atom, against the FP64 path, is
below one unit in the last place of an atom's energy (2 eV and up: 2.4e-7)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [2, 3])
def test_energy_of_a_population(tmp_path, ns):
    import maise_b200
    from maise_b200 import models, workloads

    spc = [29, 46, 47][:ns]
    ref = workloads.random_alloy(n=2, a=3.8, seed=6, jitter=0.1, species=tuple(spc))
    path = str(tmp_path / "model")
    models.random_model(path, spc, models.Basis(), (ref["X"], ref["LAT"], ref["atmn"], 3), binding=True)
    rng = np.random.default_rng(11)
    pop = []
    while len(pop) < 100:
        n = int(rng.integers(2, 40))
        L = np.eye(3) * (22.0 * n) ** (1 / 3) + rng.normal(0, 0.3, (3, 3))
        X = []
        for _ in range(20000):
            x = rng.uniform(0, 1, 3)
            d = np.array(X).reshape(-1, 3) - x
            if (np.linalg.norm((d - np.round(d)) @ L, axis=1) > 2.2).all():
                X.append(x)
            if len(X) == n:
                pop.append(dict(X=np.array(X) @ L, LAT=L, atmn=np.sort(rng.integers(0, ns, n)).astype(np.int32)))
                break
    with maise_b200.Potential(path) as pot:
        got = pot.efs_batch(pop)["H"]
        want = np.array([pot.energy(s["X"], s["LAT"], s["atmn"])["H"] for s in pop])
    nat = np.array([len(s["atmn"]) for s in pop])
    assert np.median(np.abs(want / nat)) > 2.0
    assert np.median(np.abs(got - want) / nat) < 2.4e-7
