"""Steps that stack several realizations of a small grid (chosen by the grid's
size) against one realization at a time (set_batch(1)), bit for bit: both
convolutions, both modes, grids whose noise is stacked and whose is not,
even steps with a smaller last one, repeated runs with other counts."""
import numpy as np
import pytest

from cases import bits, make_case

pytestmark = pytest.mark.gpu


def _pair(dem, streams, **kw):
    from cageo_gb300 import api
    one, many = (api.Pipeline(dem, streams, seed=9, **kw) for _ in range(2))
    one.set_batch(1)
    return one, many


def _same(one, many):
    assert np.array_equal(one.counts(), many.counts())
    for a, b in zip(one.last_stages(), many.last_stages()):
        assert np.array_equal(bits(a), bits(b))


@pytest.mark.parametrize("W,H,counts,kw", [
    (5, 4, (64, 65, 2), dict(practical_range=10.0)),
    (64, 31, (5, 5, 1, 5), {}),
    (33, 50, (3, 66), dict(use_graphs=False)),
    (257, 131, (7, 2, 7, 7), dict(filter_model=0)),
    (130, 97, (6, 4), dict(fill_mode=1)),
    (1100, 700, (67,), dict(error_stddev=0.5)),       # two steps: 34 and 33
    (1501, 1333, (35,), dict(fill_mode=1)),           # fit 33: 18 and 17
    (4200, 4100, (4, 4), {}),                         # noise slab by slab, fit 3: 2 and 2
])
def test_stacked_equals_single(cuda, W, H, counts, kw):
    dem, streams = make_case(W, H, seed=W + H, plateaus=0.1, nodata_cells=W * H // 500)
    one, many = _pair(dem, streams, **kw)
    first = 0
    for c in counts:
        one.run(first, c)
        many.run(first, c)
        first += c
        _same(one, many)
    many.close()
    one.close()


@pytest.mark.parametrize("batch", [None, 4])
def test_one_flagged_realization(cuda, batch):
    """A realization whose elevation under a stream equals NODATA is redone in
    reference order; the others of its step are not."""
    import torch
    from cageo_gb300 import api
    W, H, r = 90, 70, api.filter_radius(60.0, 10.0)
    dem, streams = make_case(W, H, seed=3)
    noise = torch.empty((H, W), device=cuda)
    api.noise_philox(noise, 9, 2, 0.0, 1.0)
    taps = api.filter_build(api.FILTER_GAUSSIAN, 60.0, 10.0, r)
    real = api.realistic_dem(torch.from_numpy(dem).to(cuda),
                             api.convolve(noise, api.FILTER_GAUSSIAN, taps, r)).cpu().numpy()
    nodata = float(real[streams >= 0][5])
    one, many = _pair(dem, streams, nodata_dem=nodata)
    if batch:
        many.set_batch(batch)
    one.run(0, 8)
    many.run(0, 8)
    _same(one, many)
    assert one.stats()["burn_reruns"] == 1 and many.stats()["burn_reruns"] == 1
    one.run(8, 8)
    many.run(8, 8)
    _same(one, many)


def test_stack_survives_save_and_tuning(cuda, tmp_path):
    """Counts saved in mid-run, other tuning and another filter in between."""
    dem, streams = make_case(200, 120, seed=8)
    one, many = _pair(dem, streams)
    for p, n in ((one, "a"), (many, "b")):
        p.run(0, 6)
        p.save(str(tmp_path / n), 6)
        p.reset_counts()
        assert p.load(str(tmp_path / n)) == 6
        p.set_tuning(64, 20)
        p.run(6, 6)
        p.run_filter(12, 6, 0, 40.0, 0.1, 2.0)
    _same(one, many)
    for p in (one, many):  # no realization: the last one's outputs stay
        p.run(18, 0)
    _same(one, many)
    for p in (one, many):
        p.profile(18)
    _same(one, many)
