"""The channel mixing and the projection sum their 64 terms in channel order, one FP32 sum
per output.  Marked gpu.

Its sums are rounded to BF16 for a whole row of the next product, so another order of the
same terms is another result: a last bit before the rounding becomes 2^-8 of a mode.  The
terms here are a large value, 62 small ones and the large one's negative, so that every
addition rounds and the order shows in whole units; everything around the mixing is exact
(powers of two, GELU at 8 and above, one retained mode), so the results are those of NumPy's
sum in order, bit for bit.
"""
import numpy as np
import pytest
import torch

from oracle import fno_oracle as fo

pytestmark = pytest.mark.gpu

L, W, M = 128, 64, 32
BATCHES = [1, 2, 8, 9, 17, 32]


def _bf16(a):
    return torch.from_numpy(np.asarray(a, dtype=np.float32)).to(torch.bfloat16).to(torch.float32).numpy()


def _terms(rng, n):
    """(n, 64) weights: 2^24, 62 values in [1, 8) and -2^24, all BF16."""
    w = _bf16(rng.uniform(1.0, 8.0, (n, W)))
    w[:, 0], w[:, -1] = 2.0 ** 24, -2.0 ** 24
    return w


def _in_order(scale, w):
    """FP32 sum of scale * w[..., v] over v in turn, one rounding a step (exact in FP64 before it)."""
    acc = np.zeros(w.shape[:-1], dtype=np.float32)
    for v in range(W):
        acc = (np.float64(scale) * w[..., v].astype(np.float64) + acc.astype(np.float64)).astype(np.float32)
    return acc


def _layer(p, l):
    o = fo.OFF_L0 + l * fo.LAYER_SIZE
    return (p[o:o + fo.LAYER_WS].reshape(W, W, M, 2), p[o + fo.LAYER_WS:o + fo.LAYER_WS + W * W].reshape(W, W),
            p[o + fo.LAYER_WS + W * W:o + fo.LAYER_SIZE])


@pytest.mark.parametrize("B", BATCHES)
def test_forward_mixing_in_channel_order(B):
    from optifax_gb300.surrogate import FNO
    rng = np.random.default_rng(B)
    p = np.zeros(fo.N_PARAMS, dtype=np.float32)
    p[fo.OFF_P:fo.OFF_PB].reshape(W, fo.CIN)[:, 4] = 1.0              # h = the conditioning channel
    w = _terms(rng, W)                                                # [output][channel]
    _layer(p, 0)[0][:, :, 0, 0] = w.T
    for l in range(1, fo.NLAYER):
        _layer(p, l)[1][:] = np.eye(W, dtype=np.float32)
    outs = [0, 21, 42, 63]
    for j, o in enumerate(outs):
        p[fo.OFF_Q:fo.OFF_QB].reshape(fo.COUT, W)[j, o] = 1.0
    scale = np.array([1.0, 2.0, 3.0, 0.5] * 8, dtype=np.float32)[:B]
    x = np.zeros((B, fo.CIN, L), dtype=np.float32)
    x[:, 4] = scale[:, None]
    net = FNO(n_bins=L, max_batch=B, params=p)
    y = net.forward(torch.from_numpy(x).to(net.dev)).cpu().numpy()
    want = np.stack([_bf16(_in_order(L * s, w[outs])) / L for s in scale])
    assert want.min() >= 8
    assert np.array_equal(y, np.broadcast_to(want[:, :, None], y.shape))


@pytest.mark.parametrize("B", BATCHES)
def test_backward_mixing_in_channel_order(B):
    from optifax_gb300.surrogate import FNO
    rng = np.random.default_rng(100 + B)
    p = np.zeros(fo.N_PARAMS, dtype=np.float32)
    w = _terms(rng, W)                                                # [input channel][output]
    _layer(p, 3)[0][:, :, 0, 0] = w
    _layer(p, 2)[2][:] = 16.0                                         # GELU and its derivative at 16: 16 and 1
    p[fo.OFF_Q:fo.OFF_QB].reshape(fo.COUT, W)[0] = 1.0
    net = FNO(n_bins=L, max_batch=B, params=p)
    x = torch.zeros((B, fo.CIN, L), device=net.dev)
    t = net.forward(x).clone()
    y0 = t[:, 0].clone()
    t[:, 0] -= 2.0 ** 24
    d = (y0 - t[:, 0]).cpu().numpy()
    assert np.all(d == d[0, 0]) and d[0, 0] > 0
    g = torch.zeros(fo.N_PARAMS, dtype=torch.float32, device=net.dev)
    net.backward(x, t, g)
    inv_n = np.float32(1.0) / np.float32(B * fo.COUT * L)
    dz = float(_bf16(np.float32(2.0) * d[0, 0] * inv_n))
    want = _bf16(_in_order(dz, w)).astype(np.float64) * (B * L)
    got = _layer(g.cpu().numpy(), 2)[2]
    assert np.array_equal(got.astype(np.float64), want)


@pytest.mark.parametrize("L_,B", [(128, 1), (192, 3), (4096, 2)])
def test_projection_in_channel_order(L_, B):
    """q, then Q_c h_c for c in turn, then the input: the output feeds the BF16 gradients of the loss."""
    from optifax_gb300.surrogate import FNO
    rng = np.random.default_rng(L_ + B)
    p = np.zeros(fo.N_PARAMS, dtype=np.float32)
    h = _bf16(rng.normal(size=W))
    _layer(p, 3)[2][:] = h
    Q = _bf16(rng.normal(size=(fo.COUT, W)))
    p[fo.OFF_Q:fo.OFF_QB] = Q.ravel()
    p[fo.OFF_QB:] = rng.normal(size=fo.COUT)
    x = rng.normal(size=(B, fo.CIN, L_)).astype(np.float32)
    net = FNO(n_bins=L_, max_batch=B, params=p)
    y = net.forward(torch.from_numpy(x).to(net.dev)).cpu().numpy()
    acc = p[fo.OFF_QB:].copy()
    for c in range(W):
        acc = (Q[:, c].astype(np.float64) * h[c] + acc.astype(np.float64)).astype(np.float32)
    assert np.array_equal(y, x[:, :fo.COUT] + acc[None, :, None])
