"""The CPU-compatible fill where the walls under water decide far and wide (no
streams, lakes over most of the grid): the wide resolution against the oracle, the
work that the resolution before it may spend, and pipelines whose steps meet such
fills unprepared."""
import numpy as np
import pytest

from cases import bits
from test_gpu_fill_bounds import fill_by_bounds

pytestmark = pytest.mark.gpu


def rough(W, H, seed=0, base=500.0, relief=10.0):
    return (np.random.default_rng(seed).random((H, W)) * relief + base).astype(np.float32)


def ridges(W, H, seed=0, base=100.0):
    y, x = np.mgrid[0:H, 0:W]
    return ((x % 64 < 2) * 50.0 + base + y * 0.001).astype(np.float32)


def holed(W, H, seed=0):
    """Rough terrain with NODATA cells, NODATA rims and cells at 0 (outlets)."""
    z = rough(W, H, seed)
    rng = np.random.default_rng(seed + 1)
    z[rng.random((H, W)) < 0.003] = -9999.0
    z[H // 3:H // 3 + 3, :W // 2] = -9999.0
    z[:, W - 1] = -9999.0
    z[rng.random((H, W)) < 2e-5] = 0.0
    return z


def stages_of(dem):
    """Filled grid and statistics of one realization without noise."""
    from cageo_gb300 import api
    p = api.Pipeline(dem, np.full(dem.shape, -9999.0, np.float32), practical_range=10.0,
                     error_stddev=0.0, seed=1)
    p.run(0, 1)
    out = p.last_stages()[0], p.stats()
    p.close()
    return out


def wide(stats):  # passes: 3 of the flood and the lists, 3 more of the wide resolution
    return stats["fill_passes"] - stats["fill_phases"] >= 6


@pytest.mark.parametrize("make,W,H", [
    (rough, 70, 90), (rough, 257, 131), (rough, 131, 257), (rough, 512, 300), (rough, 641, 511),
    (rough, 33, 2001), (rough, 2001, 33), (ridges, 320, 320), (ridges, 501, 399),
    (holed, 300, 512), (holed, 515, 389)])
def test_levels_and_work(cuda, oracle, make, W, H):
    import torch
    from cageo_gb300 import api
    dem = make(W, H)
    q, ref = oracle.pitfill(dem)
    d = torch.from_numpy(dem.copy()).cuda()
    f = api.pitfill(d)
    assert np.array_equal(bits(d.cpu().numpy()), bits(q))
    assert np.array_equal(bits(f.cpu().numpy()), bits(ref))
    if make is holed:  # (a pipeline gives such cells the noise's value)
        return
    f, stats = stages_of(dem)
    assert np.array_equal(bits(f), bits(ref))
    # Steps of a front before the fill is given up, each 3 units of work at least.
    assert stats["flood_b_passes"] <= (512 + W * H // 12000) // 3 + 1
    assert wide(stats)


@pytest.mark.parametrize("W,H,base", [(70, 90, 500.0), (150, 97, 3500.0), (257, 131, 1500.0)])
def test_phases_are_those_of_the_bounds(cuda, oracle, W, H, base):
    dem = rough(W, H, seed=3, base=base)
    q, ref = oracle.pitfill(dem)
    levels, phases = fill_by_bounds(q)
    assert np.array_equal(bits(levels.astype(np.float32)), bits(ref))
    f, stats = stages_of(dem)
    assert wide(stats) and stats["fill_phases"] == phases > 0
    assert np.array_equal(bits(f), bits(ref))


def test_static_scratch_and_workspace(cuda, oracle):
    import ctypes
    import torch
    from cageo_gb300 import api
    dem = rough(300, 517, seed=4)
    ref = oracle.pitfill(dem)[1]
    ws = torch.empty(api.lib().cageo_pitfill_workspace_size(300, 517), dtype=torch.uint8,
                     device="cuda")
    d = torch.from_numpy(dem.copy()).cuda()
    assert np.array_equal(bits(api.pitfill(d, workspace=ws).cpu().numpy()), bits(ref))
    d = torch.from_numpy(dem.copy()).cuda()
    f = torch.empty_like(d)
    torch.cuda.synchronize()
    st = api.lib().cageo_pitfill_static(ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(f.data_ptr()),
                                        300, 517, ctypes.c_float(-9999.0), 0, None)
    assert st == 0 and np.array_equal(bits(f.cpu().numpy()), bits(ref))


@pytest.mark.parametrize("batch,graphs,runs", [
    (None, True, [(0, 5)]), (None, True, [(0, 1), (1, 4)]), (None, False, [(0, 5)]),
    (1, True, [(0, 3), (3, 2)]), (1, False, [(0, 5)]), (2, True, [(0, 5)]), (2, False, [(0, 3), (3, 2)])])
def test_pipelines_meet_wide_fills(cuda, oracle, batch, graphs, runs):
    """Steps captured or not, stacked or not, with and without remainders: the
    counts are the oracle's, and the last realization's stages."""
    import torch
    from cageo_gb300 import api
    W, H = 215, 180
    dem = rough(W, H, seed=6, relief=6.0)
    streams = np.full((H, W), -9999.0, np.float32)
    p = api.Pipeline(dem, streams, practical_range=20.0, error_stddev=1.0, seed=9, use_graphs=graphs)
    if batch:
        p.set_batch(batch)
    r = api.filter_radius(20.0, 10.0)
    taps = api.filter_build(api.FILTER_GAUSSIAN, 20.0, 10.0, r)
    counts = np.zeros_like(dem)
    for k in range(5):
        noise = torch.empty((H, W), dtype=torch.float32, device="cuda")
        api.noise_philox(noise, 9, k, 0.0, 1.0)
        counts, filled, dirs, labels = oracle.realization(dem, streams, noise.cpu().numpy(), taps, r,
                                                          1, counts)
    for first, n in runs:
        p.run(first, n)
        assert wide(p.stats())
    assert np.array_equal(p.counts(), counts)
    f, d, l = p.last_stages()
    assert np.array_equal(bits(f), bits(filled))
    assert np.array_equal(d, dirs) and np.array_equal(l, labels)
    p.close()
