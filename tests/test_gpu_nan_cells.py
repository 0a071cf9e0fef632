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
