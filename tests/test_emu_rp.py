"""Host emulation of the real-plane kernels (tests/emu/emu_rp.cpp) against the oracle: their index arithmetic, barriers,
shuffles, alignment and buffer bounds, without a GPU, at sizes where they can go wrong."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import converse2d_oracle as orc
from tests.emu.build_emu import build_emu_rp

PAD = {"circular": 0, "replicate": 1, "reflect": 2, "constant": 3}
SMS = 148


@pytest.fixture(scope="module")
def emu():
    lib = ctypes.CDLL(build_emu_rp())
    lib.emu_rp_message.restype = ctypes.c_char_p
    return lib


def _ptr(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


def _check(lib, rc):
    assert rc == 0, (rc, lib.emu_rp_message())


def _weights(C, k, seed):
    rng = np.random.default_rng(seed)
    w, b = orc.init_weight(C, k, rng)
    return w, (b + rng.standard_normal(b.shape)).astype(np.float32), rng


def _forward(lib, x, w, b, s, p, mode, gelu=0, multi=0, ws_planes=0, keep=False, sms=SMS):
    """x: float32, or uint16 holding bf16"""
    B, C, H, W = x.shape
    k, bf16 = w.shape[-1], x.dtype == np.uint16
    out = np.zeros((B, C, H * s, W * s), x.dtype)
    h, wp = H + 2 * p, (W + 2 * p + 1) // 2 * 2
    r = np.zeros((B, C, h, wp), np.float32) if keep else None
    wf = np.ascontiguousarray(w.reshape(C, k, k), np.float32)
    _check(lib, lib.emu_rp_forward(_ptr(x), _ptr(out), _ptr(r), _ptr(wf), _ptr(np.ascontiguousarray(b.reshape(C))), B, C, H, W, k,
                                   s, p, PAD[mode], ctypes.c_float(1e-5), gelu, int(bf16), multi, ws_planes, sms))
    return (out, r) if keep else out


CASES = [
    # B, C, H, W, k, s, p, mode
    (1, 1, 2, 3, 1, 1, 0, "circular"),            # the smallest axes
    (1, 3, 29, 32, 3, 1, 0, "circular"),          # the largest register radices, one stage
    (2, 2, 20, 17, 5, 1, 2, "replicate"),         # 24 x 21: odd width, an unpaired column
    (1, 2, 30, 26, 3, 1, 3, "reflect"),
    (1, 1, 22, 23, 3, 1, 2, "constant"),          # 26 x 27: zero margins
    (1, 2, 33, 37, 3, 1, 0, "circular"),          # dense stages of both parities
    (1, 1, 43, 47, 3, 1, 0, "replicate"),
    (1, 1, 51, 61, 3, 1, 0, "circular"),
    (1, 1, 67, 74, 3, 1, 0, "circular"),          # 74 = 37 x 2
    (1, 1, 79, 86, 3, 1, 0, "reflect"),
    (1, 1, 111, 53, 3, 1, 1, "circular"),         # 113
    (1, 1, 53, 125, 3, 1, 1, "constant"),         # 127
    (2, 2, 16, 14, 5, 2, 2, "circular"),          # upsampling: every window, runs and bands
    (1, 2, 13, 15, 3, 3, 1, "reflect"),
    (1, 1, 10, 12, 7, 4, 3, "replicate"),
    (1, 1, 9, 11, 4, 2, 2, "constant"),           # a tap count without a compile-time epilogue
    (1, 1, 33, 35, 3, 2, 1, "circular"),          # dense stages with the epilogue
]


@pytest.mark.parametrize("case", CASES)
def test_forward_matches_the_oracle(emu, case):
    B, C, H, W, k, s, p, mode = case
    w, b, rng = _weights(C, k, H * 100 + W)
    x = rng.standard_normal((B, C, H, W)).astype(np.float32)
    ref = orc.converse2d_forward(x, w, b, s, p, mode, 1e-5, dtype=np.float64)
    outs = [_forward(emu, x, w, b, s, p, mode), _forward(emu, x, w, b, s, p, mode, multi=1, ws_planes=1 if B * C > 1 else 0)]
    for out in outs:
        assert orc.rel_l2(out, ref) <= 2e-6
    gelu = _forward(emu, x, w, b, s, p, mode, gelu=1)
    assert orc.rel_l2(gelu, torch.nn.functional.gelu(torch.from_numpy(ref)).numpy()) <= 4e-6


@pytest.mark.parametrize("H,W,sizes", [(69, 46, (128, 96)), (58, 50, (128, 192)), (29, 65, (96, 256)), (64, 23, (256, 96))])
def test_strip_block_sizes(emu, H, W, sizes):
    """Blocks of other sizes than a power of two: the last turn of a stage leaves any number of half warps without work."""
    assert tuple(emu.emu_rp_threads(2, H, W, rows, 1) for rows in (0, 1)) == sizes
    w, b, rng = _weights(2, 3, H + W)
    x = rng.standard_normal((1, 2, H, W)).astype(np.float32)
    ref = orc.converse2d_forward(x, w, b, 1, 0, "circular", 1e-5, dtype=np.float64)
    assert orc.rel_l2(_forward(emu, x, w, b, 1, 0, "circular", multi=1, sms=1), ref) <= 2e-6   # as test_forward_matches_the_oracle


FIXED = [
    # integer contractions (one SM: every tile count takes them): B, C, H, W, k, s, p, mode
    (1, 1, 132, 140, 3, 1, 1, "circular"),        # 134 x 142: the shortest axes, odd halves
    (3, 1, 130, 131, 5, 1, 2, "replicate"),       # 134 x 135: an odd width, columns alone; tiles across planes
    (1, 2, 20, 140, 3, 1, 3, "constant"),         # 26 x 146: rows alone
    (1, 1, 250, 146, 5, 1, 4, "reflect"),         # 258 x 154: one frequency and one q above 64
    (1, 1, 252, 130, 3, 1, 1, "constant"),        # 254: the longest without
    (1, 1, 32, 256, 5, 1, 6, "circular"),         # 44 x 268: four q above 64
    (1, 1, 256, 234, 7, 1, 6, "replicate"),       # 268 x 246
    (1, 2, 64, 132, 3, 2, 1, "circular"),         # 66 x 134 by 2: rows; the plane r
    (1, 1, 132, 20, 3, 3, 1, "reflect"),          # 134 x 22 by 3: columns and r
]


@pytest.mark.parametrize("case", FIXED)
def test_integer_contractions(emu, case):
    B, C, H, W, k, s, p, mode = case
    w, b, rng = _weights(C, k, H * 100 + W)
    x = rng.standard_normal((B, C, H, W)).astype(np.float32)
    ref = orc.converse2d_forward(x, w, b, s, p, mode, 1e-5, dtype=np.float64)
    out, r = _forward(emu, x, w, b, s, p, mode, multi=1, keep=True, sms=1)
    # the constants' 24 bits, two roundings of the folds and one of the result on each of four passes: 2e-7
    assert orc.rel_l2(out, ref) <= 4e-7
    gelu = _forward(emu, x, w, b, s, p, mode, gelu=1, multi=1, ws_planes=1 if B * C > 1 else 0, sms=1)
    assert orc.rel_l2(gelu, torch.nn.functional.gelu(torch.from_numpy(ref)).numpy()) <= 2e-6
    if s > 1:
        other = _forward(emu, x, w, b, s, p, mode, multi=1, keep=True)[1]
        assert orc.rel_l2(r, other) <= 2e-6


def test_integer_contractions_on_values_of_any_size(emu):
    """Lines are scaled one by one: planes of very different magnitudes, zeros, an infinity and a NaN do not meet."""
    w, b, rng = _weights(8, 3, 7)
    w[:], b[:] = w[:, :1], b[:, :1]
    x = np.repeat(rng.standard_normal((1, 1, 132, 140)).astype(np.float32), 8, axis=1)
    x[:, 6] *= np.float32(2.0 ** -100)
    x[:, 7] *= np.float32(2.0 ** -108)
    for c, f in enumerate((1.0, 2.0 ** -80, 2.0 ** 90, 0.0)):
        x[:, c] *= np.float32(f)
    x[0, 4, 60, 70], x[0, 5, 5, 9] = np.inf, np.nan
    out = _forward(emu, x, w, b, 1, 1, "circular", multi=1, sms=1)[0]
    for c, f in ((1, 2.0 ** -80), (2, 2.0 ** 90), (6, 2.0 ** -100), (7, 2.0 ** -108)):
        assert np.array_equal(out[c] / np.float32(f), out[0])      # powers of two: not one bit differs
    assert not out[3].any() and not np.isfinite(out[4]).any() and np.isnan(out[5]).all()


@pytest.mark.parametrize("case", [(1, 2, 20, 18, 3, 1, 2, "circular"), (1, 1, 21, 15, 5, 1, 2, "constant"),
                                  (1, 1, 49, 28, 3, 1, 0, "circular"), (1, 2, 11, 14, 3, 3, 1, "reflect"),
                                  (1, 2, 12, 10, 5, 2, 2, "replicate")])
def test_bf16_tensors(emu, case):
    B, C, H, W, k, s, p, mode = case
    w, b, rng = _weights(C, k, H + W)
    x = torch.from_numpy(rng.standard_normal((B, C, H, W)).astype(np.float32)).bfloat16()
    ref = orc.converse2d_forward(x.float().numpy(), w, b, s, p, mode, 1e-5, dtype=np.float64)
    bits = x.view(torch.int16).numpy().view(np.uint16)
    for multi in (0, 1):
        out = _forward(emu, bits, w, b, s, p, mode, multi=multi)
        got = torch.from_numpy(out.view(np.int16)).view(torch.bfloat16).float().numpy()
        assert orc.rel_l2(got, ref) <= 3e-3


@pytest.mark.parametrize("case", [
    (2, 2, 14, 17, 3, 1, 3, "replicate"),
    (3, 1, 20, 15, 5, 1, 2, "reflect"),
    (2, 1, 12, 12, 3, 1, 8, "circular"),        # margins almost as wide as the plane
    (2, 2, 10, 14, 5, 2, 2, "circular"),
    (2, 1, 9, 12, 7, 3, 3, "reflect"),
    (1, 2, 8, 7, 3, 4, 1, "constant"),
    (2, 1, 8, 9, 4, 3, 2, "replicate"),         # run-time taps and scale
    (2, 1, 14, 39, 3, 1, 1, "circular"),        # 41: dense stage along x
])
def test_gradient_kernels_match_fp64_autograd(emu, case):
    from conversenet_b200.autograd import spectral_forward
    B, C, H, W, k, s, p, mode = case
    w, b, rng = _weights(C, k, H * W)
    x = rng.standard_normal((B, C, H, W)).astype(np.float32)
    g = rng.standard_normal((B, C, H * s, W * s)).astype(np.float32)
    out, r = _forward(emu, x, w, b, s, p, mode, keep=True)
    h, wd = H + 2 * p, W + 2 * p
    nseg, hh = (2 if B > 1 else 1), h // 2 + 1
    gx, D, taps = np.zeros_like(x), np.zeros((C, wd, hh, 2), np.float32), np.zeros((B, C, k, k), np.float32)
    wf, bf = np.ascontiguousarray(w.reshape(C, k, k)), np.ascontiguousarray(b.reshape(C))
    _check(emu, emu.emu_rp_backward(_ptr(x), _ptr(g), _ptr(r), _ptr(gx), _ptr(D), _ptr(taps), _ptr(wf), _ptr(bf), B, C, H, W, k, s,
                                    p, PAD[mode], ctypes.c_float(1e-5), nseg, SMS))
    X, Wt, Bt = (torch.from_numpy(a).double().requires_grad_(True) for a in (x, w, b))
    y = spectral_forward(X, Wt, Bt, s, p, mode, 1e-5)
    ref, = torch.autograd.grad(y, X, torch.from_numpy(g).double())
    assert orc.rel_l2(gx, ref.numpy()) <= 2e-6
    # D = 4 sum_b FFT2(pad(x_b)) conj(FFT2(q_b)): q is the extended cotangent, at scale >= 2 its strided correlation
    from conversenet_b200.autograd import _Cotangent, _pad
    cot = _Cotangent(torch.from_numpy(g), torch.from_numpy(wf), k, s, p)
    q = (cot.g_full if s == 1 else cot.v).double()
    d = (torch.fft.fft2(_pad(torch.from_numpy(x).double(), p, mode)) * torch.fft.fft2(q).conj()).sum(0)[:, :hh]
    got = torch.view_as_complex(torch.from_numpy(D).double()).transpose(1, 2) / 4
    assert float((got - d).abs().pow(2).sum().sqrt() / d.abs().pow(2).sum().sqrt()) <= 2e-6
    if s > 1:
        full, rr = cot.g_full.double(), torch.from_numpy(r[..., :wd]).double()
        for a in range(k):
            for c in range(k):
                moved = torch.roll(full, (a - k // 2, c - k // 2), (-2, -1))[..., ::s, ::s]
                want, most = (moved * rr).sum((-2, -1)), moved.norm(dim=(-2, -1)) * rr.norm(dim=(-2, -1))
                # r itself is within 1e-6 of its norm; a sum that cancels has no relative error to speak of
                assert bool((torch.from_numpy(taps[:, :, a, c]).double() - want).abs().le(2e-6 * most).all())


@pytest.mark.parametrize("case", [
    # integer contractions (one SM: every tile count takes them): columns of a zero-extended or strided cotangent, rows with
    # the conjugated multiplier (dL/dx alone: the parameters' rows have a kernel of their own), columns back without a crop
    (1, 1, 132, 140, 3, 1, 1, "circular"),        # 134 x 142
    (2, 1, 130, 131, 5, 1, 2, "replicate"),       # 134 x 135: columns alone; tiles across planes
    (1, 1, 20, 134, 3, 1, 0, "circular"),         # rows alone, no padding
    (1, 1, 256, 140, 5, 1, 1, "reflect"),         # 258 x 142: one q above 64
    (1, 1, 128, 264, 3, 1, 2, "constant"),        # 132 x 268: four q above 64
    (1, 1, 132, 32, 3, 2, 1, "circular"),         # 134 x 34 by 2
])
@pytest.mark.parametrize("params", [False, True])
def test_gradients_through_the_integer_contractions(emu, case, params):
    from conversenet_b200.autograd import _Cotangent, _pad, spectral_forward
    B, C, H, W, k, s, p, mode = case
    w, b, rng = _weights(C, k, H * W)
    x = rng.standard_normal((B, C, H, W)).astype(np.float32)
    g = rng.standard_normal((B, C, H * s, W * s)).astype(np.float32)
    r = _forward(emu, x, w, b, s, p, mode, keep=True, multi=1, sms=1)[1]
    h, wd = H + 2 * p, W + 2 * p
    hh = h // 2 + 1
    gx, D, taps = np.zeros_like(x), np.zeros((C, wd, hh, 2), np.float32) if params else None, np.zeros((B, C, k, k), np.float32)
    wf, bf = np.ascontiguousarray(w.reshape(C, k, k)), np.ascontiguousarray(b.reshape(C))
    _check(emu, emu.emu_rp_backward(_ptr(x), _ptr(g), _ptr(r), _ptr(gx), _ptr(D), _ptr(taps), _ptr(wf), _ptr(bf), B, C, H, W, k, s,
                                    p, PAD[mode], ctypes.c_float(1e-5), 1, 1))
    X, Wt, Bt = (torch.from_numpy(a).double().requires_grad_(True) for a in (x, w, b))
    ref, = torch.autograd.grad(spectral_forward(X, Wt, Bt, s, p, mode, 1e-5), X, torch.from_numpy(g).double())
    # test_integer_contractions' bound; the padding's adjoint and the correlation add a few fp32 sums
    assert orc.rel_l2(gx, ref.numpy()) <= 6e-7
    if not params:
        return
    cot = _Cotangent(torch.from_numpy(g), torch.from_numpy(wf), k, s, p)
    q = (cot.g_full if s == 1 else cot.v).double()
    d = (torch.fft.fft2(_pad(torch.from_numpy(x).double(), p, mode)) * torch.fft.fft2(q).conj()).sum(0)[:, :hh]
    got = torch.view_as_complex(torch.from_numpy(D).double()).transpose(1, 2) / 4
    assert float((got - d).abs().pow(2).sum().sqrt() / d.abs().pow(2).sum().sqrt()) <= 2e-6


def test_routes_and_shared_memory(emu):
    one = lambda n, planes: emu.emu_rp_one_block(1, planes, n, n, 1, 0, SMS)
    assert [one(76, 64), one(108, 1), one(110, 98), one(110, 99), one(132, 99), one(132, 64)] == [1, 1, 0, 1, 1, 0]
    assert [one(96, 149), one(98, 149), one(136, 148), one(140, 148), one(74, 10)] == [1, 0, 1, 0, 0]     # 74: dense stage
    r0, r1 = ctypes.c_int(), ctypes.c_int()
    for n in range(2, 1400):
        width = emu.emu_rp_plan(n, ctypes.byref(r0), ctypes.byref(r1))
        if width < 0:
            continue
        assert r0.value * r1.value == n and r0.value <= 127 and r1.value <= 26 and (width == 0 or r1.value <= 16)
        assert emu.emu_rp_fits(n, n, 1, SMS) == 1 and emu.emu_rp_fits(n, n, 1000, SMS) == 1
