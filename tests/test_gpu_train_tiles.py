"""Training objective and gradient where the tiles of the forward and gradient
kernels end: species of 0, 1, 8, 9 and past 128 atoms, input counts that are no
multiple of 4 or 64, layers of 1 to 32 units, with and without force terms.
Held to the CPU oracle by the bar of the training tests: 1e-12 of the largest
component (1e-11 with forces), sums of at most a few hundred terms."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.train import objective

pytestmark = pytest.mark.gpu

SPC = [29, 46, 47]


@pytest.mark.parametrize("forces", [False, True])
@pytest.mark.parametrize("counts,h", [
    ((5,), (10, 10)), ((1, 9), (1, 1)), ((8, 0, 17), (17, 5)), ((129, 1, 70), (10, 10)), ((128, 127), (16, 32)),
    ((33, 264), (32, 17)),
])
def test_tiles(tmp_path, counts, h, forces):
    from maise_b200 import models, workloads
    from maise_b200.train import Trainer

    ns = len(counts)
    rng = np.random.default_rng(sum(counts) + h[0])
    ref = workloads.random_alloy(n=2, a=3.7, seed=6, species=SPC[:ns], jitter=0.1)
    path = str(tmp_path / "model")
    models.random_model(path, SPC[:ns], models.Basis(), (ref["X"], ref["LAT"], ref["atmn"], 3), h=h, seed=3)
    t = models.read_model(path)
    spc = rng.permutation(np.repeat(np.arange(ns), counts)).astype(np.int32)
    Na = len(spc)
    nat = np.array([5] * (Na // 5) + ([Na % 5] if Na % 5 else []), np.int32)
    X = rng.uniform(0, 1, (Na, t["arch"][0]))
    G = t["rmin"][spc] + X / t["dr"][spc]
    X = (G - t["rmin"][spc]) * t["dr"][spc]
    E = -3.0 * nat + rng.normal(0, 1, len(nat))
    w = rng.uniform(0.5, 1.5, len(nat))
    tr = Trainer(path, None, E, weights=w, WE=1.3, LREG=1e-5, descriptors=(G, spc, nat))
    fd = None
    if forces:
        first = np.concatenate([[0], np.cumsum(nat)])
        pick = rng.integers(0, len(nat), 6)
        own = [first[s] + rng.permutation(nat[s]) for s in pick]
        off = np.concatenate([[0], np.cumsum([len(o) for o in own])])
        fd = dict(f_atom=np.array([o[0] for o in own]), F_ref=rng.normal(0, 1, (6, 3)), blk_off=off,
                  blk_atom=np.concatenate(own), Fn=rng.normal(0, 0.1, (off[-1], t["arch"][0], 3)), WF=0.6)
        tr.set_forces(fd["f_atom"], fd["F_ref"], off, fd["blk_atom"], fd["Fn"], WF=0.6, scale_blocks=False)
    V = tr.initial()
    RT, g, Ep = tr.eval(V)
    tr.close()
    RTo, go, Eo = objective(V, X, spc, nat, E, w, 1.3, 1e-5, ns, *t["arch"][1:], forces=fd)
    assert RT == pytest.approx(RTo, rel=1e-11)
    np.testing.assert_allclose(Ep, Eo, rtol=1e-12, atol=1e-12)
    np.testing.assert_allclose(g, go, rtol=0, atol=(1e-11 if forces else 1e-12) * np.abs(go).max())
