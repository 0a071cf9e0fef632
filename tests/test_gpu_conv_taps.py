"""The separable convolution's loop over taps: every remainder of a group of 8,
fewer taps than a group, and the largest radii, on grids of a few tiles, against
the oracle bit for bit; the fused front takes the same loop in a pipeline."""
import numpy as np
import pytest

from cases import bits, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [0, 1, 2, 3, 4, 5, 6, 7, 8, 11, 12, 14, 22, 24, 30, 40, 63, 88])
def test_taps(cuda, oracle, r):
    import torch
    from cageo_gb300 import api
    rng = np.random.default_rng(r)
    taps = rng.standard_normal(2 * r + 1).astype(np.float32)
    for W, H in ((r + 1, r + 3), (131, 97), (204, 90)):
        if r >= min(W, H):
            continue
        f = rng.standard_normal((H, W)).astype(np.float32)
        got = api.convolve(torch.from_numpy(f).to(cuda), api.FILTER_GAUSSIAN, taps, r)
        assert np.array_equal(bits(got.cpu().numpy()), bits(oracle.convolve(f, taps, r, 1))), (W, H)


@pytest.mark.parametrize("r,tile", [(9, 0), (30, 1), (40, 3), (64, 2)])
def test_front(cuda, oracle, r, tile):
    import torch
    from cageo_gb300 import api
    W, H = 190, 143
    dem, streams = make_case(W, H, seed=r)
    cut = r * 4.0 - 1.0  # metres: the practical range of this radius at 10 m cells
    assert api.filter_radius(cut, 10.0) == r
    p = api.Pipeline(dem, streams, practical_range=cut, error_stddev=1.0, seed=2)
    p.set_tuning(64, 20, tile)
    p.run(0, 1)
    noise = torch.empty((H, W), dtype=torch.float32, device=cuda)
    api.noise_philox(noise, 2, 0, 0.0, 1.0)
    taps = api.filter_build(api.FILTER_GAUSSIAN, cut, 10.0, r)
    counts, filled, dirs, labels = oracle.realization(dem, streams, noise.cpu().numpy(), taps, r, 1,
                                                      np.zeros_like(dem))
    assert np.array_equal(p.counts(), counts)
    assert np.array_equal(bits(p.last_stages()[0]), bits(filled))
    p.close()
