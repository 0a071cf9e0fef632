"""The short forms of the stages' roundings -- quantization without a division,
diagonal drops by a multiplication and a correction -- against IEEE arithmetic
(numpy's float32), over every index and every mantissa; and the fused front's
quick path against the oracle."""
import numpy as np
import pytest

from cases import bits, make_case

pytestmark = pytest.mark.gpu
F = np.float32


def test_quantization_of_every_index(cuda):
    """Every millimetre below 4000 m (and some above, where the short form ends)
    and the floats next to it on either side: truncation of 1000 e, at least 1,
    over 1000."""
    import torch
    from cageo_gb300 import api
    k = np.arange(1, 4000000 + 96, dtype=np.int64)
    e = (k / 1000).astype(F)
    e = np.stack([np.nextafter(e, F(0)), e, np.nextafter(e, F(np.inf))], 1).reshape(-1)
    W = 4096
    e = np.concatenate([e, np.full(-e.size % W, 4000.0, F)]).reshape(-1, W)
    index = np.maximum(np.trunc(F(1000) * e), F(1))
    want = index / F(1000)
    assert index.dtype == F and want.dtype == F
    v = torch.from_numpy(e).to(cuda)
    api.pitfill(v)  # quantizes its input in place
    assert np.array_equal(bits(v.cpu().numpy()), bits(want))


def test_quantization_of_small_values(cuda):
    import torch
    from cageo_gb300 import api
    rng = np.random.default_rng(3)
    e = np.exp(rng.uniform(np.log(1e-44), np.log(1.0), (512, 512))).astype(F)
    e[0, :4] = [0.0, 1e-45, 0.001, 3999.9999]
    index = np.where(e == 0, F(0), np.maximum(np.trunc(F(1000) * e), F(1)))
    v = torch.from_numpy(e).to(cuda)
    api.pitfill(v)
    assert np.array_equal(bits(v.cpu().numpy()), bits(index / F(1000)))


def _diagonal_drops(cuda, x):
    """Routing of cells with a drop of x to the north-east and, to the north, one
    of x / sqrt 2 (first maximum: north) or of the float below it (north-east)."""
    import torch
    from cageo_gb300 import api
    y = x / F(1.41421356237309505)
    assert y.dtype == F
    n = int(x.size ** 0.5)
    for drop, want in ((y, (0, -1)), (np.nextafter(y, F(0)), (1, -1))):
        dem = torch.ones((4 * n, 4 * n), device=cuda)
        dem[1::4, 1::4] = 1e-42  # differences to it are the drops themselves
        dem[0::4, 1::4] = -torch.from_numpy(drop.reshape(n, n)).to(cuda)
        dem[0::4, 2::4] = -torch.from_numpy(x.reshape(n, n)).to(cuda)
        d = api.route_d8(dem)[1::4, 1::4]
        assert bool((d[..., 0] == want[0]).all()) and bool((d[..., 1] == want[1]).all())


def test_diagonal_drop_of_every_mantissa(cuda):
    for base in range(0x3f800000, 0x40800000, 1 << 20):  # the floats of [1, 4)
        _diagonal_drops(cuda, np.arange(base, base + (1 << 20), dtype=np.uint32).view(F))


@pytest.mark.parametrize("lo,hi", [(-114, -90), (-101, -98), (-98, 98), (98, 101), (98, 126)])
def test_diagonal_drop_over_the_exponents(cuda, lo, hi):
    """Across the limits of the short form's range (1e-30 and 1e30) and beyond."""
    rng = np.random.default_rng(hi - lo)
    m = rng.uniform(1.0, 2.0, 1 << 18).astype(F)
    _diagonal_drops(cuda, np.ldexp(m, rng.integers(lo, hi + 1, 1 << 18)).astype(F))


@pytest.mark.parametrize("W", [64, 68, 75])
@pytest.mark.parametrize("lo,hi,nodata", [(80.0, 180.0, -9999.0), (-4.0, 4.0, -9999.0), (3990.0, 4010.0, -9999.0),
                                          (0.0, 0.01, -9999.0), (80.0, 180.0, 100.0), (80.0, 180.0, 9999.0)])
def test_front_against_the_oracle(cuda, oracle, W, lo, hi, nodata):
    """The pipeline's filled grid against the oracle's fill of the burned grid
    that the stage calls give: quads with NODATA, streams, bevels, cells pushed
    below 0, above 4000 and to the limits of the range."""
    import torch
    from cageo_gb300 import api
    H = 70
    rng = np.random.default_rng(int(lo) + W + 1)
    _, streams = make_case(W, H, seed=W)
    dem = rng.uniform(lo, hi, (H, W)).astype(F)
    dem[rng.random((H, W)) < 0.02] = nodata
    r = api.filter_radius(60.0, 10.0)
    taps = api.filter_build(api.FILTER_GAUSSIAN, 60.0, 10.0, r)
    noise = torch.empty((H, W), dtype=torch.float32, device=cuda)
    for mode in (api.FILL_CPU_COMPAT, api.FILL_EXACT):
        p = api.Pipeline(dem, streams, error_stddev=1.5, seed=21, nodata_dem=nodata, fill_mode=mode)
        p.set_batch(1)
        p.run(0, 2)
        f = p.last_stages()[0]
        p.close()
        api.noise_philox(noise, 21, 1, 0.0, 1.5)
        field = api.convolve(noise, api.FILTER_GAUSSIAN, taps, r).cpu().numpy()
        burned = oracle.stream_burn(oracle.realistic_dem(dem, field, nodata), streams,
                                    nodata_dem=nodata)
        want = (oracle.pitfill_exact(burned, nodata) if mode == api.FILL_EXACT
                else oracle.pitfill(burned, nodata)[1])
        assert np.array_equal(bits(f), bits(want))
