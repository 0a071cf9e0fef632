"""Many resolutions of small grids, four streams at once: every grid-wide wait
ends, and the counts are those of the same jobs one after another."""
import numpy as np
import pytest

from cases import make_case

pytestmark = pytest.mark.gpu


def test_many_concurrent_jobs(cuda):
    from cageo_gb300 import batch
    grids = [make_case(W, H, seed=W, pits=W * H // 150) for W, H in
             [(600, 500), (257, 613), (900, 300), (1200, 101)]]
    b = batch.Batch(grids, seed=5)
    jobs = batch.mixed_jobs(4, 1000, 5, range_m=(30.0, 60.0))
    b.run(jobs)
    many = b.counts()
    for p in b.pipes:
        p.reset_counts()
    b.run(jobs, concurrent=False)
    for x, y in zip(many, b.counts()):
        assert np.array_equal(x, y)
    b.close()
