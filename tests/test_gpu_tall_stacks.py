"""Batched steps of a grid so tall that a whole batch has more rows of tiles
than a launch may: the steps hold fewer realizations, the results are the
single ones."""
import numpy as np
import pytest

from cases import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,batch,count", [(65535, 64, 64), (40000, 64, 55), (32768, 64, 3)])
def test_batch_of_tall_grids(cuda, H, batch, count):
    from cageo_gb300 import api
    W = 8
    rng = np.random.default_rng(H)
    dem = rng.uniform(80.0, 90.0, (H, W)).astype(np.float32)
    streams = np.where(rng.random((H, W)) < 0.01, np.float32(1), np.float32(-9999))
    one, many = (api.Pipeline(dem, streams, practical_range=10.0, seed=3) for _ in range(2))
    one.set_batch(1)
    many.set_batch(batch)
    one.run(0, count)
    many.run(0, count)
    assert np.array_equal(one.counts(), many.counts())
    for a, b in zip(one.last_stages(), many.last_stages()):
        assert np.array_equal(bits(a), bits(b))
    one.close()
    many.close()
