"""Surrogate kernels at the edges of their tiles: layer tiles of 128 bins cut by 64, batches
on both sides of the mixing kernel's eight, envelope transforms of every radix remainder,
and an output that lies over its input.  Marked gpu.
"""
import numpy as np
import pytest
import torch

from oracle import fno_oracle as fo

pytestmark = pytest.mark.gpu

# as in the network's oracle test: activations in BF16, 4 layers
Y_TOL, G_TOL = 2e-2, 5e-2


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("L,B", [(192, 2), (192, 9), (320, 8), (128, 17)])
def test_network_at_cut_tiles_and_mixed_batches(L, B):
    from optifax_gb300.gemm import tc_error
    from optifax_gb300.surrogate import FNO, init_params
    rng = np.random.default_rng(7 * L + B)
    p = init_params(3, spec_scale=8.0)
    x = rng.normal(size=(B, fo.CIN, L)).astype(np.float32)
    t = rng.normal(size=(B, fo.COUT, L)).astype(np.float32)
    net = FNO(n_bins=L, max_batch=B, params=p)
    xg, tg = torch.from_numpy(x).to(net.dev), torch.from_numpy(t).to(net.dev)
    g = torch.zeros(fo.N_PARAMS, dtype=torch.float32, device=net.dev)
    y = net.forward(xg).cpu().numpy()
    net.backward(xg, tg, g)
    g = g.cpu().numpy()
    assert tc_error() == 0
    _, gref, yref = fo.loss_and_grads(p, x, t, weights_bf16=True)
    assert _rel(y, yref) <= Y_TOL
    cuts = [fo.OFF_P, fo.OFF_PB]
    for l in range(fo.NLAYER):
        o = fo.OFF_L0 + l * fo.LAYER_SIZE
        cuts += [o, o + fo.LAYER_WS, o + fo.LAYER_WS + 4096]
    cuts += [fo.OFF_Q, fo.OFF_QB, fo.N_PARAMS]
    for a, b in zip(cuts[:-1], cuts[1:]):
        assert _rel(g[a:b], gref[a:b]) <= G_TOL, (a, b)


def test_output_over_the_input():
    """The C entry writes y over x (one sample's x is 6 rows, its y 4) after x is read."""
    from optifax_gb300 import _native as nat
    from optifax_gb300.surrogate import FNO, init_params
    L, B = 128, 3
    net = FNO(n_bins=L, max_batch=B, params=init_params(4))
    x = torch.from_numpy(np.random.default_rng(2).normal(size=(B, 6, L)).astype(np.float32)).to(net.dev)
    want = net.forward(x).clone()
    st = int(torch.cuda.current_stream(net.dev).cuda_stream)
    nat.check(nat.load().optifax_fno_forward(net.h, x.data_ptr(), x.data_ptr(), B, st), None, "fno_forward")
    got = x.reshape(-1)[:B * 4 * L].reshape(B, 4, L)
    # split sums change their order from run to run: FP32 rounding, then BF16 activations
    assert _rel(got.cpu().numpy(), want.cpu().numpy()) <= Y_TOL


@pytest.mark.parametrize("L", [2, 4, 8, 16, 32, 64, 512, 1024, 2048, 4096])
def test_envelope_transforms_of_every_length(L):
    """Against NumPy's FP64 transform.  log2 L stages of a few 6e-8 each, and sigma's and
    the scale's rounding: below 5e-6 at 4096."""
    from optifax_gb300 import fastforward as ff
    N = L + 3 * (L // 2) + 1
    kc_p, kc_s = N - 1, L // 2
    lo, hi = -(L // 2), max(L // 4, 1) if L > 2 else 1
    crop = ff.EnvCrop(N, L, (kc_p, lo, hi, kc_s, lo, hi), 0.75)
    rng = np.random.default_rng(L)
    Y = (rng.normal(size=(3, N)) + 1j * rng.normal(size=(3, N))).astype(np.complex64)
    x, sig = ff.encode(torch.from_numpy(Y).cuda(), crop)
    x, sig = x.cpu().numpy().astype(np.float64), sig.cpu().numpy().astype(np.float64)
    for p in range(3):
        ep = ff.envelope(Y[p].astype(np.complex128), kc_p, lo, hi, L)
        es = ff.envelope(Y[p].astype(np.complex128), kc_s, lo, hi, L)
        s = np.sqrt(np.mean(np.abs(es) ** 2))
        assert abs(sig[p] - s) <= 5e-6 * s
        assert _rel(x[p, 0] + 1j * x[p, 1], ep / crop.pump_scale) <= 5e-6
        assert _rel(x[p, 2] + 1j * x[p, 3], es / s) <= 5e-6
    # the inverse, with the bins outside the bands cleared; disjoint bands
    hi_d = max(hi - 1, lo + 1)
    crop = ff.EnvCrop(N, L, (N - 1, lo, hi_d, (N - 1 + hi_d - lo) % N, lo, hi_d), 0.75)
    y = rng.normal(size=(1, 4, L)).astype(np.float32)
    sg = torch.tensor([1.5], device="cuda")
    out = torch.full((N,), 7.0 + 1j, dtype=torch.complex64, device="cuda")
    X = ff.decode_env(crop, torch.from_numpy(y).cuda(), sg, X_out=out).cpu().numpy()
    ref = np.zeros(N, dtype=np.complex128)
    for b, scale in ((0, 0.75), (1, 1.5)):
        e = np.fft.fft(y[0, 2 * b].astype(np.float64) + 1j * y[0, 2 * b + 1]) / L * scale
        kc, lo_, hi_ = crop.band[3 * b:3 * b + 3]
        o = np.arange(lo_, hi_)
        ref[(kc + o) % N] = e[o % L]
    assert _rel(X, ref) <= 5e-6
    assert np.all(X[ref == 0] == 0)


@pytest.mark.parametrize("N,ldc,shift", [(64, 64, 0), (64, 65, 0), (64, 68, 1), (72, 72, 0)])
def test_split_sums_off_16_bytes(N, ldc, shift):
    """Split sums by 16-byte reductions, and element-wise where C's rows or its base are not
    on 16 bytes or a tile is cut; the tolerance is test_gemm_gpu.py's."""
    from optifax_gb300.gemm import gemm_bf16, tc_error
    g = torch.Generator().manual_seed(N + ldc + shift)
    M, K = 200, 512
    A = torch.randn(256, K, generator=g).to(torch.bfloat16).cuda()
    B = torch.randn(128, K, generator=g).to(torch.bfloat16).cuda()
    buf = torch.zeros(M * ldc + shift, device="cuda")
    C = buf[shift:].view(M, ldc)[:, :N]
    gemm_bf16(A, B, C, M=M, N=N, splits=4)
    assert tc_error() == 0
    R = A[:M].float() @ B[:N].float().T
    assert (C - R).abs().max().item() / R.abs().max().item() < 1e-5
    if ldc > N:
        assert bool((buf[shift:].view(M, ldc)[:, N:] == 0).all()) and bool((buf[:shift] == 0).all())
