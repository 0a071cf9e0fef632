"""Training on grids a few cells wide, on both sides of the lines where a cell a
thread (12 columns) and a block per channel pair (24 columns; cells x columns up
to 65536) give way to tiles: against float64 sums, with the bounds of the tiles'
test; infinite values stay where they are terms."""
import numpy as np
import pytest

import cnn_oracle as co
from test_gpu_train_tiles import EPS, _bf16, _conv, _cuda, _params, _wgrad, test_training_tiles

pytestmark = pytest.mark.gpu
_check = test_training_tiles
del test_training_tiles  # (its own cases run in its own file)


@pytest.mark.parametrize("W,H,B", [(1, 300, 4), (3, 401, 2), (3, 7282, 1), (6, 5, 9), (12, 37, 3),
                                   (12, 455, 1), (12, 456, 1), (13, 37, 3), (24, 113, 1),
                                   (24, 114, 1), (25, 9, 2)])
def test_training(cuda, W, H, B):
    _check(cuda, W, H, B)


@pytest.mark.parametrize("W", [5, 12, 24])
def test_infinite_values(cuda, W):
    """An infinite weight of the upper left tap and an infinite activation under a
    zero gradient."""
    import torch
    from cageo_gb300 import api
    H, B = 11, 2
    rng = np.random.default_rng(W)
    p, layers = _params(W)
    feat = np.abs(rng.standard_normal((B, 4, H, W))).astype(np.float32)
    layers[1][0][5, 7, 0] = np.inf
    a1, a2, out = (t.cpu().numpy() for t in api.ws_forward(_cuda(p), _cuda(feat)))
    ref, mag = _conv(a1, _bf16(layers[1][0]), _bf16(layers[1][1]))
    fin = np.isfinite(ref)
    assert fin[:, 5, 0].all() and fin[:, 5, :, 0].all() and np.array_equal(fin, fin & np.isfinite(a2))
    assert (np.abs(a2 - np.maximum(ref, 0))[fin] <= 289 * EPS * mag[fin]).all()
    p, layers = _params(W + 1)
    a1, a2 = (np.abs(rng.standard_normal((B, 32, H, W))).astype(np.float32) for _ in range(2))
    dy = rng.standard_normal((B, H, W)).astype(np.float32)
    dy[1, 4:7, 1:4] = 0
    a2[1, 3, 5, 2] = np.inf
    g = torch.zeros(co.N_PARAMS, device=cuda)
    api.ws_backward(_cuda(p), _cuda(feat), _cuda(a1), _cuda(a2), _cuda(dy), g)
    g3 = g.cpu().numpy()[10432:10720].reshape(1, 32, 9)
    ref, mag = _wgrad(dy[:, None], a2)
    assert np.isfinite(ref).all() and np.isfinite(g3).all()
    assert (np.abs(g3 - ref) <= (W * H * B + 20) * EPS * mag).all()
