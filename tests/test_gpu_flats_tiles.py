"""Routing of flats where the tile flood can go wrong: large level areas that
cross many tiles, exits and layers on tile rims and corners, grids at tile
edges, unaligned grids, NODATA among the levels, both rule sets.  Bit-exact
against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 40), (31, 33), (32, 32), (33, 31), (64, 96), (65, 63), (200, 37), (300, 260)]


def _levels(W, H, seed, levels, nodata):
    """Few distinct levels in blocks: flats everywhere, some without an exit."""
    rng = np.random.default_rng(seed)
    k = max(1, int(rng.integers(3, 45)))
    coarse = rng.integers(1, levels + 1, (H // k + 2, W // k + 2)).astype(np.float32)
    dem = np.repeat(np.repeat(coarse, k, 0), k, 1)[:H, :W].copy()
    dem[rng.random((H, W)) < 0.002] = 0.0
    dem[rng.random((H, W)) < 0.01] -= 0.5
    if nodata:
        dem[rng.random((H, W)) < 0.01] = -9999.0
    return dem


@pytest.mark.parametrize("levels,nodata", [(2, False), (6, False), (4, True)])
@pytest.mark.parametrize("W,H", SIZES)
def test_flats_at_tile_edges(cuda, oracle, W, H, levels, nodata):
    import torch
    from cageo_gb300 import api
    for seed in (1, 2):
        dem = _levels(W, H, seed * 100 + W + H, levels, nodata)
        # 4 bytes past a 16-byte boundary for one of the seeds
        buf = torch.empty(W * H + 1, dtype=torch.float32, device=cuda)
        v = buf[seed - 1:seed - 1 + W * H].view(H, W)
        v.copy_(torch.from_numpy(dem))
        d, fd = api.route_d8(v, with_flatdist=True)
        assert np.array_equal(d.cpu().numpy(), oracle.flow_route(dem))
        assert np.array_equal(api.route_d8(v).cpu().numpy(), d.cpu().numpy())
        g, gfd = api.route_d8(v, with_flatdist=True, mode=api.ROUTE_GPU_ORDER)
        gr, gfr = oracle.flow_route_gpu(dem, with_flatdist=True)
        assert np.array_equal(g.cpu().numpy(), gr)
        assert np.array_equal(gfd.cpu().numpy(), gfr)
        # The CPU rules' distances: the same layers where no NODATA cell and
        # no stream is near.
        if not nodata:
            assert np.array_equal(fd.cpu().numpy() > 1, gfr > 1)


def test_long_flat_and_steep_diagonals(cuda, oracle):
    """A level corridor winding over many tiles (distances far beyond one
    segment of levels), and drops whose diagonal quotients tie or nearly tie."""
    import torch
    from cageo_gb300 import api
    H, W = 190, 330
    dem = np.full((H, W), 9.0, np.float32)
    for k, y in enumerate(range(5, H - 5, 4)):
        dem[y, 5:W - 5] = 3.0
        x = W - 6 if k % 2 == 0 else 5
        dem[y:y + 5, x] = 3.0
    dem[1:6, 5] = 2.0
    d, fd = api.route_d8(torch.from_numpy(dem).to(cuda), with_flatdist=True)
    assert np.array_equal(d.cpu().numpy(), oracle.flow_route(dem))
    assert int(fd.max()) > 4000
    rng = np.random.default_rng(8)
    base = rng.choice(np.float32([1.0, 1.4142135, 1.4142137, 2.0, 2.828427, 2.8284273, 1e-20, 3e38]),
                      (97, 131)).astype(np.float32)
    t = torch.from_numpy(base).to(cuda)
    assert np.array_equal(api.route_d8(t).cpu().numpy(), oracle.flow_route(base))
