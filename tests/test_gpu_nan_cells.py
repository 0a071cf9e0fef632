"""Grids that hold NaN (and infinite) elevations, stage by stage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _flats(W, H, seed):
    """Few levels in blocks, with NaN cells inside the flats, in lines that cut
    them in two, and on the rims and corners of the 32x32 tiles."""
    rng = np.random.default_rng(seed)
    k = int(rng.integers(5, 40))
    coarse = rng.integers(1, 4, (H // k + 2, W // k + 2)).astype(np.float32)
    dem = np.repeat(np.repeat(coarse, k, 0), k, 1)[:H, :W].copy()
    dem[rng.random((H, W)) < 0.003] -= 0.5
    dem[rng.random((H, W)) < 0.001] = 0.0
    dem[rng.random((H, W)) < 0.004] = np.inf
    dem[rng.random((H, W)) < 0.002] = -np.inf
    dem[rng.random((H, W)) < 0.01] = np.nan
    dem[H // 2, 1:W - W // 3] = np.nan
    dem[:, W // 2][rng.random(H) < 0.7] = np.nan
    for y in (0, 31, 32, 63, 64):
        for x in (0, 31, 32, 63, 64):
            if y < H and x < W and rng.random() < 0.5:
                dem[y, x] = np.nan
    return dem


@pytest.mark.parametrize("W,H", [(9, 9), (33, 32), (64, 64), (70, 97), (257, 131)])
def test_routing_through_nan_cells(cuda, oracle, W, H):
    """CPU rules: no direction for a NaN cell inside a flat, and no path through
    it.  GPU order: elevations count in layer 1 only."""
    import torch
    from cageo_gb300 import api
    for seed in (1, 2, 3):
        dem = _flats(W, H, seed)
        if W == 9:
            dem[:], dem[4, 4] = 5.0, np.nan
        v = torch.from_numpy(dem).to(cuda)
        d, fd = api.route_d8(v, with_flatdist=True)
        assert np.array_equal(d.cpu().numpy(), oracle.flow_route(dem))
        inner = np.isnan(dem)
        inner[0] = inner[-1] = inner[:, 0] = inner[:, -1] = False
        assert (fd.cpu().numpy()[inner] == 0).all()
        g, gfd = api.route_d8(v, with_flatdist=True, mode=api.ROUTE_GPU_ORDER)
        gr, gfr = oracle.flow_route_gpu(dem, with_flatdist=True)
        assert np.array_equal(g.cpu().numpy(), gr)
        assert np.array_equal(gfd.cpu().numpy(), gfr)


def _exact_fill(dem, nodata=-9999.0):
    """The exact fill's levels by relaxation: a NaN elevation bounds no level
    (the larger of it and a level is the level), and a NaN outlet passes none on."""
    H, W = dem.shape
    keep = (dem == nodata) | (dem == 0)
    keep[0] = keep[-1] = keep[:, 0] = keep[:, -1] = True
    w = np.where(keep, dem, np.float32(np.inf))
    while True:
        r = np.pad(np.where((dem == nodata) | np.isnan(w), np.float32(np.inf), w), 1,
                   constant_values=np.inf)
        m = np.full_like(w, np.inf)
        for dy in range(3):
            for dx in range(3):
                if (dy, dx) != (1, 1):
                    m = np.minimum(m, r[dy:dy + H, dx:dx + W])
        n = np.where(keep, dem, np.minimum(w, np.fmax(dem, m)))
        if np.array_equal(n, w, equal_nan=True):
            return np.where(~keep & np.isinf(n), np.float32(99990000.0), n)
        w = n


@pytest.mark.parametrize("W,H", [(12, 9), (33, 32), (65, 70), (130, 97)])
def test_exact_fill_with_nan_cells(cuda, W, H):
    """NaN outlets (a border of them, as a frame without data leaves) pass no
    level on from one neighbour to another; NaN cells inside do."""
    import torch
    from cageo_gb300 import api
    for seed in range(4):
        rng = np.random.default_rng(seed * 100 + W)
        dem = rng.uniform(1.0, 9.0, (H, W)).astype(np.float32)
        frame = np.zeros((H, W), bool)
        frame[0] = frame[-1] = frame[:, 0] = frame[:, -1] = True
        dem[frame & (rng.random((H, W)) < (0.9 if seed % 2 else 0.4))] = np.nan
        dem[rng.random((H, W)) < 0.02] = np.nan
        dem[rng.random((H, W)) < 0.01] = -9999.0
        dem[0, 0] = 1.0
        want = _exact_fill(dem)
        v = torch.from_numpy(dem).to(cuda)
        f = api.pitfill(v.clone(), mode=api.FILL_EXACT).cpu().numpy()
        assert np.array_equal(f, want, equal_nan=True)
        warm = torch.full_like(v, float("inf"))
        f = api.pitfill_exact_warm(v, warm)
        f = (f[0] if isinstance(f, tuple) else f).cpu().numpy()
        assert np.array_equal(f, want, equal_nan=True)
