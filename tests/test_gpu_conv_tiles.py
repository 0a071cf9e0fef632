"""The convolutions where their tiles can go wrong: radii around the padding to
16 bytes and the switch of the 2D kernel's staging, odd and tiny grids, every
wrap, unaligned grids.  Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(5, 4), (64, 32), (65, 33), (132, 71), (200, 260), (1027, 130)])
@pytest.mark.parametrize("model,r", [(1, 0), (1, 1), (1, 3), (1, 7), (1, 13), (1, 15), (1, 16), (1, 23), (1, 61),
                                     (0, 0), (0, 1), (0, 4), (0, 19), (0, 31), (0, 32), (0, 64)])
def test_convolution_tiles(cuda, oracle, W, H, model, r):
    import torch
    from cageo_gb300 import api
    if r >= min(W, H):
        pytest.skip("the radius must be below the grid size")
    rng = np.random.default_rng(r * 1000 + W)
    x = rng.standard_normal((H, W)).astype(np.float32)
    L = 2 * r + 1
    taps = rng.standard_normal(L if model == 1 else L * L).astype(np.float32)
    want = oracle.convolve(x, taps, r, model)
    for off in (0, 1):  # and 4 bytes past a 16-byte boundary
        buf = torch.empty(W * H + 1, dtype=torch.float32, device=cuda)
        v = buf[off:off + W * H].view(H, W)
        v.copy_(torch.from_numpy(x))
        got = api.convolve(v, model, taps, r).cpu().numpy()
        assert np.array_equal(got.view(np.int32), want.view(np.int32))


def test_largest_radius_still_fits(cuda):
    """The largest radii the kernels took before are still taken, the next ones
    still refused."""
    import torch
    from cageo_gb300 import api
    x = torch.zeros((200, 200), device=cuda)
    for model, ok, bad in ((1, 88, 89), (0, 72, 73)):
        n = 2 * ok + 1
        api.convolve(x, model, np.zeros(n if model else n * n, np.float32), ok)
        n += 2
        with pytest.raises(api.CageoError):
            api.convolve(x, model, np.zeros(n if model else n * n, np.float32), bad)
