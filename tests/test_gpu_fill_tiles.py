"""The pit fill where its tiles, rims, work queue and resolution lists can go
wrong: grids at tile edges and a few cells wide, areas no outlet reaches,
terrain with many non-passable cells (large pockets, several phases), and
workspaces left over from other fills.  Bit-exact against the oracle."""
import numpy as np
import pytest

from cases import bits, make_case

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 2), (3, 1), (1, 40), (5, 3), (31, 33), (32, 32), (33, 31), (64, 64), (65, 63),
         (96, 40), (3, 2000), (2000, 3), (129, 257)]


def _terrain(kind, W, H, seed):
    """fbm: rounded terrain; rough: random levels in lakes of pits; high: the
    same near 3000 m, where a quarter of the 1 mm levels is non-passable;
    islands: NODATA frames around areas without an outlet."""
    rng = np.random.default_rng(seed)
    if kind == "fbm" and min(W, H) >= 16:
        return make_case(W, H, seed=seed, pits=max(W * H // 200, 1))[0]
    base = 3000.0 if kind == "high" else 20.0
    dem = (base + rng.uniform(0.0, 1.0, (H, W)) ** 2 * (0.4 if kind == "high" else 4.0)).astype(np.float32)
    if kind == "islands":
        dem[rng.random((H, W)) < 0.02] = -9999.0
        for _ in range(max(1, W * H // 4000)):
            y, x = int(rng.integers(0, H)), int(rng.integers(0, W))
            h, w = int(rng.integers(3, 80)), int(rng.integers(3, 80))
            dem[y:y + h, x] = dem[y:y + h, min(x + w, W - 1)] = -9999.0
            dem[y, x:x + w] = dem[min(y + h, H - 1), x:x + w] = -9999.0
        dem[rng.random((H, W)) < 0.001] = 0.0
    return dem


@pytest.mark.parametrize("kind", ["fbm", "rough", "high", "islands"])
@pytest.mark.parametrize("W,H", SIZES)
def test_fill_at_tile_edges(cuda, oracle, kind, W, H):
    import torch
    from cageo_gb300 import api
    dem = _terrain(kind, W, H, seed=W * 7 + H)
    q_ref, f_ref = oracle.pitfill(dem)
    v = torch.from_numpy(dem.copy()).to(cuda)
    f = api.pitfill(v)
    assert np.array_equal(bits(v.cpu().numpy()), bits(q_ref))
    assert np.array_equal(bits(f.cpu().numpy()), bits(f_ref))
    e = api.pitfill(torch.from_numpy(dem).to(cuda), mode=api.FILL_EXACT)
    assert np.array_equal(bits(e.cpu().numpy()), bits(oracle.pitfill_exact(dem)))


@pytest.mark.parametrize("kind,W,H", [("rough", 700, 500), ("high", 700, 500), ("islands", 900, 700)])
def test_fill_with_many_pockets(cuda, oracle, kind, W, H):
    """Pockets by the thousand: long lists, reopened components, phases --
    into a workspace full of another fill's remains."""
    import torch
    from cageo_gb300 import api
    ws = torch.full((api.lib().cageo_pitfill_workspace_size(W, H),), 0xFF, dtype=torch.uint8,
                    device=cuda)
    for seed in (1, 2):
        dem = _terrain(kind, W, H, seed=seed)
        _, f_ref = oracle.pitfill(dem)
        f = api.pitfill(torch.from_numpy(dem).to(cuda), workspace=ws)
        assert np.array_equal(bits(f.cpu().numpy()), bits(f_ref))


@pytest.mark.parametrize("warps,rounds", [(16, 1), (20, 2), (22, 64)])
def test_pipeline_fill_at_every_setting(cuda, oracle, warps, rounds):
    """The flood's block sizes and a visit's round limit (a capped visit queues
    its own tile), on a stack whose slabs straddle tiles."""
    from cageo_gb300 import api
    dem, streams = make_case(150, 77, seed=9, pits=200)
    p = api.Pipeline(dem, streams, error_stddev=1.5, seed=4)
    p.run(0, 6)
    want = p.counts()
    p.reset_counts()
    p.set_batch(3)
    p.set_tuning(rounds, warps)
    p.run(0, 6)
    assert np.array_equal(p.counts(), want)


def test_batched_only_pipeline_reports_its_own_status(cuda):
    """A pipeline that has run batched steps only, in memory that was used
    before: the status words of its single-step workspaces were never written
    and are not errors."""
    import torch
    from cageo_gb300 import api
    dem, streams = make_case(400, 300, seed=3)
    junk = [torch.full((1 << 22,), -1, dtype=torch.int32, device=cuda) for _ in range(8)]
    del junk
    torch.cuda.empty_cache()
    p = api.Pipeline(dem, streams, error_stddev=1.5, seed=4)
    p.set_batch(4)
    p.run(0, 4)
    one = api.Pipeline(dem, streams, error_stddev=1.5, seed=4)
    one.run(0, 4)
    assert np.array_equal(p.counts(), one.counts())


@pytest.mark.parametrize("n", [60, 600])
def test_basin_behind_one_wall_cell(cuda, oracle, n):
    """A flat basin that drains through a single non-passable cell of a flooded
    tunnel: the resolution lowers n x n cells from one entry, in steps that
    outgrow its buffers."""
    import torch
    from cageo_gb300 import api
    k = np.arange(2001, 4000)
    q = (k / 1000).astype(np.float32)
    wall = q[np.trunc(np.float32(1000) * q) < k][0]
    dem = np.full((n + 40, n + 30), 100.0, np.float32)
    dem[0] = dem[-1] = dem[:, 0] = dem[:, -1] = 1.0
    dem[0, 0] = 0.0
    dem[20, 1], dem[20, 2:10], dem[20, 10] = 20.0, 2.0, wall
    dem[15:15 + n, 11:11 + n] = 10.0
    _, f_ref = oracle.pitfill(dem)
    assert f_ref[300 if n == 600 else 40, 40] == 20.0
    f = api.pitfill(torch.from_numpy(dem).to(cuda))
    assert np.array_equal(bits(f.cpu().numpy()), bits(f_ref))
