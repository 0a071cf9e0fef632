"""The training kernels at the edges of their tiles (32 columns, 4 and 8 rows),
unaligned rows and batches, against float64 sums with the error bound of
float32 summation; infinite values, which padding and cells without gradient
must not spread."""
import numpy as np
import pytest

import cnn_oracle as co

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _bf16(x):
    u = np.ascontiguousarray(x, np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000
    return u.astype(np.uint32).view(np.float32).astype(np.float64)


def _taps(H, W):
    """(tap, output slices, input slices) of a zero-padded 3x3 window."""
    for t in range(9):
        dy, dx = t // 3 - 1, t % 3 - 1
        o = (slice(max(0, -dy), H - max(0, dy)), slice(max(0, -dx), W - max(0, dx)))
        i = (slice(max(0, dy), H - max(0, -dy)), slice(max(0, dx), W - max(0, -dx)))
        yield t, o, i


def _conv(x, w, bias):
    """Sums and sums of magnitudes of a convolution, padding left out."""
    B, cin, H, W = x.shape
    x = x.astype(np.float64)
    out = np.zeros((B, w.shape[0], H, W)) + bias[:, None, None]
    mag = np.abs(out)
    for t, o, i in _taps(H, W):
        p = w[None, :, :, t, None, None] * x[(slice(None), None, slice(None)) + i]
        out[(slice(None), slice(None)) + o] += p.sum(2)
        mag[(slice(None), slice(None)) + o] += np.abs(p).sum(2)
    return out, mag


def _wgrad(dz, a):
    B, cin, H, W = a.shape
    dz, a = dz.astype(np.float64), a.astype(np.float64)
    g = np.zeros((dz.shape[1], cin, 9))
    m = np.zeros_like(g)
    for t, o, i in _taps(H, W):
        d = dz[(slice(None), slice(None), None) + o]
        with np.errstate(invalid="ignore"):
            p = np.where(d == 0, 0.0, d * a[(slice(None), None) + (slice(None),) + i])
        g[:, :, t] = p.sum((0, 3, 4))
        m[:, :, t] = np.abs(p).sum((0, 3, 4))
    return g, m


def _params(seed):
    p = (np.random.default_rng(seed).standard_normal(co.N_PARAMS) * 0.2).astype(np.float32)
    return p, [(p[0:1152].reshape(32, 4, 9), p[1152:1184]),
               (p[1184:10400].reshape(32, 32, 9), p[10400:10432]),
               (p[10432:10720].reshape(1, 32, 9), p[10720:])]


def _flip(w):
    return w.transpose(1, 0, 2)[:, :, ::-1]


def _cuda(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()


@pytest.mark.parametrize("W,H,B", [(1, 1, 1), (2, 3, 2), (4, 4, 1), (31, 9, 1), (32, 8, 3), (33, 5, 2),
                                   (36, 7, 1), (64, 64, 2), (70, 37, 3), (8, 130, 5), (200, 96, 2)])
def test_training_tiles(cuda, W, H, B):
    import torch
    from cageo_gb300 import api
    rng = np.random.default_rng(W * 100 + H)
    p, layers = _params(W + H)
    feat = rng.standard_normal((B, 4, H, W)).astype(np.float32)
    a1, a2, out = (t.cpu().numpy() for t in api.ws_forward(_cuda(p), _cuda(feat)))
    x = feat
    for k, got in enumerate((a1, a2, out[:, None])):
        w, b = layers[k]
        ref, mag = _conv(x, _bf16(w), _bf16(b))
        if k < 2:
            ref = np.maximum(ref, 0)
        assert (np.abs(got - ref) <= (9 * x.shape[1] + 1) * EPS * mag).all()
        x = got
    dy = rng.standard_normal((B, H, W)).astype(np.float32)
    dy[rng.random(dy.shape) < 0.3] = 0
    grad = np.ones(co.N_PARAMS, np.float32)
    g = _cuda(grad)
    tmp1, tmp2 = (torch.empty((B, 32, H, W), device=cuda) for _ in range(2))
    api.ws_backward(_cuda(p), _cuda(feat), _cuda(a1), _cuda(a2), _cuda(dy), g, tmp1, tmp2)
    g = g.cpu().numpy().astype(np.float64) - 1
    # The input gradients in float64; their own float32 error is covered by
    # the bound's second term.
    n = W * H * B
    zero = np.zeros(32)
    d3 = dy[:, None].astype(np.float64)
    d2 = _conv(d3, _flip(_bf16(layers[2][0])), zero)
    d1 = _conv(d2[0] * (a2 > 0), _flip(_bf16(layers[1][0])), zero)
    d1m = _conv(d2[1] * (a2 > 0), np.abs(_flip(_bf16(layers[1][0]))), zero)[0]
    for lo, mid, hi, dz, mag, a, chain in (
            (10432, 10720, 10721, d3, np.abs(d3), a2, 0),
            (1184, 10400, 10432, d2[0] * (a2 > 0), d2[1] * (a2 > 0), a1, 10),
            (0, 1152, 1184, d1[0] * (a1 > 0), d1m * (a1 > 0), feat, 300)):
        ref, _ = _wgrad(dz, a)
        _, m = _wgrad(mag, np.abs(a))
        tol = (n + chain + 20) * EPS
        assert (np.abs(g[lo:mid].reshape(ref.shape) - ref) <= tol * (m + 1)).all(), lo
        assert (np.abs(g[mid:hi] - dz.sum((0, 2, 3))) <= tol * (mag.sum((0, 2, 3)) + 1)).all(), lo


def test_infinite_weight_does_not_reach_past_the_edge(cuda):
    """An infinite weight of the upper left tap: the first row and column, where
    it meets padding, stay finite (as sums that leave the padding out)."""
    from cageo_gb300 import api
    p, layers = _params(3)
    feat = np.abs(np.random.default_rng(0).standard_normal((1, 4, 9, 40))).astype(np.float32)
    layers[1][0][5, 7, 0] = np.inf
    layers[2][0][0, 5, 0] = np.inf
    a1, a2, out = (t.cpu().numpy() for t in api.ws_forward(_cuda(p), _cuda(feat)))
    assert np.isfinite(a1).all()
    ref, mag = _conv(a1, _bf16(layers[1][0]), _bf16(layers[1][1]))
    fin = np.isfinite(ref)
    assert fin[:, 5, 0].all() and fin[:, 5, :, 0].all() and not fin[:, 5, 1:, 1:].all()
    ok = fin & np.isfinite(a2)
    assert np.array_equal(fin, ok)
    assert (np.abs(a2 - np.maximum(ref, 0))[ok] <= 289 * EPS * mag[ok]).all()
    with np.errstate(invalid="ignore"):
        ref3, _ = _conv(a2, _bf16(layers[2][0]), _bf16(layers[2][1]))
    assert np.array_equal(np.isfinite(ref3[:, 0]), np.isfinite(out))


@pytest.mark.parametrize("where", ["activation", "gradient"])
def test_infinite_value_in_weight_gradients(cuda, where):
    """An infinite activation under a zero gradient, or an infinite gradient in
    a corner: only the sums that it is a term of are affected."""
    import torch
    from cageo_gb300 import api
    H, W, B = 21, 45, 2
    rng = np.random.default_rng(1)
    p, layers = _params(5)
    feat = rng.standard_normal((B, 4, H, W)).astype(np.float32)
    a1, a2 = (np.abs(rng.standard_normal((B, 32, H, W))).astype(np.float32) for _ in range(2))
    dy = rng.standard_normal((B, H, W)).astype(np.float32)
    if where == "activation":
        dy[1, 8:13, 28:33] = 0
        a2[1, 3, 10, 30] = np.inf
    else:
        dy[0, 0, 0] = np.inf
    g = torch.zeros(co.N_PARAMS, device=cuda)
    api.ws_backward(_cuda(p), _cuda(feat), _cuda(a1), _cuda(a2), _cuda(dy), g)
    g3 = g.cpu().numpy()[10432:10720].reshape(1, 32, 9)
    ref, mag = _wgrad(dy[:, None], a2)
    ok = np.isfinite(ref)
    assert ok.any() and np.array_equal(ok, np.isfinite(g3))
    assert (np.abs(g3 - ref)[ok] <= (W * H * B + 20) * EPS * mag[ok]).all()
