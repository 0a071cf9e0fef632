"""The CPU-compatible fill of terrain without streams, where lakes without an
outlet leave most cells to the resolution: the levels against the oracle, and
the work of the resolution (its confirmation phases) against a plain restatement
of the bounds that it may use."""
import numpy as np
import pytest

from cases import bits

pytestmark = pytest.mark.gpu
INF = np.float32(np.inf)


def _neighbours(a, fill):
    p = np.pad(a, 1, constant_values=fill)
    H, W = a.shape
    return [p[dy:dy + H, dx:dx + W] for dy in range(3) for dx in range(3) if (dy, dx) != (1, 1)]


def _relax(level, q, relay, fixed):
    """max(q, least relayed level of the neighbours) until no level falls."""
    while True:
        m = np.minimum.reduce(_neighbours(np.where(relay(level), level, INF), INF))
        n = np.where(fixed, level, np.minimum(level, np.maximum(q, m)))
        if np.array_equal(n, level):
            return level
        level = n


def _components(mask):
    from scipy.ndimage import label
    return label(mask, np.ones((3, 3), int))[0]


def fill_by_bounds(q):
    """(levels, phases) of the quantized grid q without NODATA and zeros."""
    least = q.min()
    index = np.trunc(np.float32(1000) * (q - least))
    passable = index / np.float32(1000) + least == q
    border = np.ones(q.shape, bool)
    border[1:-1, 1:-1] = False
    wall = ~passable & ~border
    start = np.where(border, q, INF)
    s = _relax(start, q, lambda v: passable, border)
    a = _relax(s, q, lambda v: passable | (wall & (s > q)), border)
    part = _components(a != s)
    reopened = np.unique(part[wall & (s > q) & (a <= q)])
    opened = np.isin(part, reopened[reopened > 0])
    sure = wall & (a > q) & (s > q)  # expands in every case
    confirmed = sure.copy()
    relay = lambda v: passable | (confirmed & (v > q))
    level = _relax(np.where(opened, s, a), q, relay, border)
    part = _components(opened & (level != a))
    phases = 0
    while True:
        pending = (part > 0) & wall & ~confirmed & (level > q)
        reached = pending & (level < INF)
        if not reached.any():
            return np.where(level == INF, q, level), phases
        phases += 1
        m = np.full(part.max() + 1, INF)
        np.minimum.at(m, part[reached], level[reached])
        confirmed |= pending & (q <= m[part]) & (m[part] < INF)
        level = _relax(level, q, relay, border)


def terrain(W, H, base, seed):
    """Hills of a few metres around bowls, rounded to 1 mm by the fill."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:H, 0:W]
    z = rng.uniform(0.0, 0.3, (H, W))
    for _ in range(W * H // 900):
        r, cy, cx = rng.uniform(4, 22), rng.uniform(0, H), rng.uniform(0, W)
        z -= rng.uniform(0.5, 3.0) * np.maximum(0.0, 1.0 - np.hypot(y - cy, x - cx) / r)
    return (z - z.min() + base).astype(np.float32)


@pytest.mark.parametrize("W,H,base", [(60, 50, 1.0), (120, 90, 1500.0), (150, 130, 2500.0),
                                      (131, 97, 3500.0), (200, 170, 600.0)])
def test_phases_are_those_of_the_bounds(cuda, oracle, W, H, base):
    from cageo_gb300 import api
    seen = 0
    for seed in range(4):
        dem = terrain(W, H, base, seed)
        q, ref = oracle.pitfill(dem)
        levels, phases = fill_by_bounds(q)
        assert np.array_equal(bits(levels.astype(np.float32)), bits(ref))
        p = api.Pipeline(dem, np.full((H, W), -9999.0, np.float32), practical_range=10.0,
                         error_stddev=0.0, seed=1)
        p.run(0, 1)
        f = p.last_stages()[0]
        stats = p.stats()
        p.close()
        assert np.array_equal(bits(f), bits(ref))
        assert stats["fill_phases"] == phases
        seen += phases
    assert seen > 0
