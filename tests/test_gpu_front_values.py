"""The fused front's quick path for four ordinary cells at once against the
oracle: quads that hold NODATA, streams, bevels, cells pushed below 0, above
4000 and to the limits of the range, and NODATA values inside it."""
import numpy as np
import pytest

from cases import bits, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [64, 68, 75])
@pytest.mark.parametrize("lo,hi,nodata", [(80.0, 180.0, -9999.0), (-4.0, 4.0, -9999.0), (3990.0, 4010.0, -9999.0),
                                          (0.0, 0.01, -9999.0), (80.0, 180.0, 100.0), (80.0, 180.0, 9999.0)])
def test_front_values(cuda, oracle, W, lo, hi, nodata):
    import torch
    from cageo_gb300 import api
    H = 70
    rng = np.random.default_rng(int(lo) + W)
    _, streams = make_case(W, H, seed=W)
    dem = rng.uniform(lo, hi, (H, W)).astype(np.float32)
    dem[rng.random((H, W)) < 0.02] = nodata
    r = api.filter_radius(60.0, 10.0)
    taps = api.filter_build(api.FILTER_GAUSSIAN, 60.0, 10.0, r)
    noise = torch.empty((H, W), dtype=torch.float32, device=cuda)
    for mode in (api.FILL_CPU_COMPAT, api.FILL_EXACT):
        p = api.Pipeline(dem, streams, error_stddev=1.5, seed=21, nodata_dem=nodata, fill_mode=mode)
        p.set_batch(1)
        p.run(0, 2)
        f, d, lab = p.last_stages()
        api.noise_philox(noise, 21, 1, 0.0, 1.5)
        v = api.convolve(noise, api.FILTER_GAUSSIAN, taps, r)
        v = api.realistic_dem(torch.from_numpy(dem).to(cuda), v, nodata)
        api.stream_burn(v, torch.from_numpy(streams).to(cuda), nodata_dem=nodata)
        want = api.pitfill(v, nodata_dem=nodata, mode=mode).cpu().numpy()
        assert np.array_equal(bits(f), bits(want))
