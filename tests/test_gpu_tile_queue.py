"""The asynchronous tile queue of the pit fill's flood and of the flat search:
tiles handed from one SM to another, their results bit-exact against the
oracle however the visits fall."""
import numpy as np
import pytest

from cases import bits

pytestmark = pytest.mark.gpu


def _corridor(W, H, seed):
    """A channel one cell wide winding through high ground from an outlet at 1:
    every tile on its way is visited again and again."""
    rng = np.random.default_rng(seed)
    dem = rng.uniform(200.0, 300.0, (H, W)).astype(np.float32)
    dem[0] = dem[-1] = dem[:, 0] = dem[:, -1] = 400.0
    for k, y in enumerate(range(2, H - 3, 2)):
        dem[y, 2:W - 2] = rng.uniform(2.0, 90.0, W - 4).astype(np.float32)
        x = W - 3 if k % 2 == 0 else 2
        dem[y + 1, x] = rng.uniform(2.0, 90.0)
    dem[0, 2], dem[1, 2] = 1.0, 2.0
    return dem


@pytest.mark.parametrize("W,H", [(96, 96), (131, 75), (330, 190)])
def test_levels_and_distances_across_tiles(cuda, oracle, W, H):
    """Row lengths that are no multiple of a tile put cells of two tiles into one
    cache line; a visit must see what the tile's last visit, on another SM,
    wrote."""
    import torch
    from cageo_gb300 import api
    dem = _corridor(W, H, seed=W)
    _, f_ref = oracle.pitfill(dem)
    e_ref = oracle.pitfill_exact(dem)
    d_ref = oracle.flow_route(e_ref)
    v = torch.from_numpy(dem).to(cuda)
    e_dev = torch.from_numpy(e_ref).to(cuda)
    for _ in range(5):
        assert np.array_equal(bits(api.pitfill(v.clone()).cpu().numpy()), bits(f_ref))
        e = api.pitfill(v.clone(), mode=api.FILL_EXACT)
        assert np.array_equal(bits(e.cpu().numpy()), bits(e_ref))
        assert np.array_equal(api.route_d8(e_dev).cpu().numpy(), d_ref)


def test_many_short_drains(cuda, oracle):
    """Grids of a few tiles, where most warps wait with a ticket while the last
    tiles are pushed: every drain ends, with nothing left behind."""
    import torch
    from cageo_gb300 import api
    for W, H in [(33, 64), (70, 70), (100, 40)]:
        dem = _corridor(W, H, seed=W)
        e_ref = oracle.pitfill_exact(dem)
        d_ref = torch.from_numpy(oracle.flow_route(e_ref)).to(cuda)
        e_dev = torch.from_numpy(e_ref).to(cuda)
        v = torch.from_numpy(dem).to(cuda)
        for _ in range(200):
            assert torch.equal(api.pitfill(v, mode=api.FILL_EXACT), e_dev)
            assert torch.equal(api.route_d8(e_dev), d_ref)


def test_tiles_queued_while_processed(cuda):
    """One sweep round per visit: nearly every visit ends with its tile queued
    again, by itself and by its neighbours."""
    from cageo_gb300 import api
    from cases import make_case
    dem, streams = make_case(257, 131, seed=5, pits=400)
    p = api.Pipeline(dem, streams, error_stddev=1.5, seed=4)
    p.run(0, 200)
    want = p.counts()
    for warps in (16, 22):
        p.reset_counts()
        p.set_tuning(1, warps)
        p.run(0, 200)
        assert np.array_equal(p.counts(), want)
    p.close()
