"""Host threads that each use their own handle, or the RDF call, at different
histogram sizes: the shared-memory limit of a kernel is a setting that they
share, so it may not follow one call's size."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(jobs):
    failed = []

    def body(job):
        try:
            job()
        except Exception as e:  # the assertion below shows it
            failed.append(repr(e))

    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def _structure():
    rng = np.random.default_rng(1)
    return [dict(X=rng.uniform(0, 6, (6, 3)), LAT=6.0 * np.eye(3), atmn=np.zeros(6, np.int32))]


def test_surrogates_of_different_histograms():
    from maise_b200.surrogate import Surrogate

    s = _structure()

    def job(nspc, nbins):
        def run():
            sur = Surrogate(nspc, nbins=nbins)
            first = sur.features(s)
            for _ in range(2000):
                last = sur.features(s)
            np.testing.assert_allclose(last, first, rtol=1e-5, atol=1e-6 * np.abs(first).max())
            sur.close()

        return run

    _run([job(1, 1400), job(1, 2000), job(1, 3000), job(2, 1800)])


def test_rdfs_of_different_sizes():
    from maise_b200 import evos

    s = _structure()

    def job(nspc, nbins):
        def run():
            first = evos.rdf(s, nspc, nbins=nbins)
            for _ in range(300):
                last = evos.rdf(s, nspc, nbins=nbins)
            np.testing.assert_allclose(last, first, rtol=1e-12, atol=1e-13)

        return run

    _run([job(1, 6000), job(2, 3000), job(3, 3000), job(3, 4000)])
