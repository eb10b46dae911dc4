"""The real-plane kernels (`csrc/cvb_rp.cuh`: run-time two-stage plans, one plane at a time), their gradients and the
block kernels around them, at the sizes where they can go wrong: every width of the dense large-prime stage at its
smallest and largest length, one-stage axes, odd and even lengths, strips and bands with remainders."""
import numpy as np
import pytest
import torch

from oracle import converse2d_oracle as orc

pytestmark = pytest.mark.gpu


def _rel(a, r):
    return float((a.detach().double() - r.double()).norm() / r.double().norm())


CASES = [
    # B, C, H, W, k, s, p, mode, dtype
    (1, 1, 2, 3, 1, 1, 0, "circular", "fp32"),            # the smallest axes
    (1, 3, 29, 32, 3, 1, 0, "circular", "fp32"),          # largest register radices, one stage
    (1, 2, 37, 41, 3, 1, 0, "replicate", "fp32"),         # dense stage, width 20: both ends
    (1, 2, 43, 47, 5, 1, 0, "reflect", "fp32"),           # width 24
    (3, 2, 53, 61, 3, 1, 0, "constant", "fp32"),          # width 32
    (1, 2, 67, 73, 7, 1, 0, "circular", "fp32"),          # width 36
    (1, 2, 79, 89, 3, 1, 0, "circular", "fp32"),          # width 44
    (1, 2, 97, 113, 3, 1, 0, "circular", "fp32"),         # widths 56 and 64
    (1, 2, 127, 254, 3, 1, 0, "circular", "fp32"),
    (2, 3, 131 * 2 - 2, 53 * 12 - 2, 3, 1, 1, "replicate", "fp32"),   # 262 is refused below; 636 = 53 * 12
    (1, 130, 20, 26, 3, 1, 2, "constant", "bf16"),        # one block a plane, constant margins
    (2, 5, 26 * 26 - 4, 40, 3, 1, 2, "circular", "fp32"),   # 676 = 26 * 26
    (1, 3, 77, 118, 3, 3, 1, "reflect", "bf16"),          # epilogue through a band, ragged rows
    (2, 70, 19, 23, 5, 3, 2, "replicate", "fp32"),
    (1, 2, 33, 301, 3, 4, 1, "constant", "bf16"),         # bands shorter than a row segment
    (1, 2, 21, 18, 4, 2, 2, "circular", "fp32"),          # tap count without a compile-time epilogue
    (1, 2, 24, 27, 3, 5, 1, "circular", "fp32"),          # scale without one
    (3, 4, 128, 128, 5, 2, 4, "circular", "fp32"),        # odd batch at a size with pair kernels
]


@pytest.mark.parametrize("case", CASES)
def test_forward_matches_oracle(case):
    from conversenet_b200 import Converse2D
    B, C, H, W, k, s, p, mode, dt = case
    rng = np.random.default_rng(H * 1000 + W)
    w, b = orc.init_weight(C, k, rng)
    b = b + rng.standard_normal(b.shape).astype(np.float32)
    dtype = torch.float32 if dt == "fp32" else torch.bfloat16
    x = torch.from_numpy(rng.standard_normal((B, C, H, W)).astype(np.float32)).to(dtype)
    m = Converse2D(C, C, k, scale=s, padding=p, padding_mode=mode).cuda().eval()
    with torch.no_grad():
        m.weight.copy_(torch.from_numpy(w))
        m.bias.copy_(torch.from_numpy(b))
        if (H + 2 * p) % 131 == 0:
            with pytest.raises(RuntimeError):      # a prime factor above 127
                m(x.cuda())
            return
        y = m(x.cuda()).float().cpu().numpy()
    ref = orc.converse2d_forward(x.float().numpy(), w, b, s, p, mode, 1e-5, dtype=np.float64)
    assert orc.rel_l2(y, ref) <= (2e-6 if dt == "fp32" else 3e-3)


@pytest.mark.parametrize("case", [
    # integer contractions: enough planes that they are taken on the largest chips; a few planes are compared
    (1, 176, 132, 140, 3, 1, 1, "circular", "fp32"),      # 134 x 142: the shortest
    (2, 64, 252, 156, 5, 1, 1, "constant", "fp32"),       # 254 x 158: columns too long for one more q
    (1, 96, 256, 240, 7, 1, 6, "replicate", "bf16"),      # 268 x 252: four q above 64; bf16 columns
    (3, 40, 250, 232, 3, 1, 4, "reflect", "fp32"),        # 258 x 240
    (1, 80, 40, 256, 3, 1, 6, "circular", "fp32"),        # 52 x 268: rows alone
    (1, 70, 242, 243, 3, 2, 1, "circular", "fp32"),       # 244 x 245 by 2: an odd width
    (1, 3, 200, 192, 3, 1, 1, "circular", "fp32"),        # 202 x 194: wide dense stages, any number of planes
])
def test_integer_contractions(case):
    from conversenet_b200 import Converse2D, _cabi
    B, C, H, W, k, s, p, mode, dt = case
    rng = np.random.default_rng(H * 1000 + W)
    w, b = orc.init_weight(C, k, rng)
    b = b + rng.standard_normal(b.shape).astype(np.float32)
    dtype = torch.float32 if dt == "fp32" else torch.bfloat16
    x = torch.from_numpy(rng.standard_normal((B, C, H, W)).astype(np.float32)).to(dtype)
    m = Converse2D(C, C, k, scale=s, padding=p, padding_mode=mode).cuda().eval()
    with torch.no_grad():
        m.weight.copy_(torch.from_numpy(w))
        m.bias.copy_(torch.from_numpy(b))
        y = m(x.cuda()).float().cpu().numpy()
    some = sorted({0, C // 2, C - 1})
    ref = orc.converse2d_forward(x.float().numpy()[-1:, some], np.ascontiguousarray(w[:, some]), np.ascontiguousarray(b[:, some]),
                                 s, p, mode, 1e-5, dtype=np.float64)
    # fp32: see tests/test_emu_rp.py; at scale 2 the epilogue's sums of nine come on top
    assert orc.rel_l2(y[-1:, some], ref) <= (4e-7 if dt == "fp32" else 3e-3)
    assert _cabi.load().cvb_last_device_status(1) == 0      # no bounded wait has run out


def test_a_table_of_another_batch_is_refused():
    """The real-plane table that one image reads is not what full pairs of planes of 268 x 268 read."""
    from conversenet_b200 import Converse2D
    from conversenet_b200 import functional as CF
    m = Converse2D(64, 64, 3, padding=6, padding_mode="circular").cuda()
    table, wf = CF.build_transfer(m.weight, m.bias, 1, 1e-5, 268, 268, batch=1)
    for B in (2, 8):                # (from 128 planes on the modules themselves keep that table)
        with pytest.raises(RuntimeError, match="another batch size"):
            CF.converse2d_forward(torch.randn(B, 64, 256, 256, device="cuda"), table, wf, 3, 1, 6, "circular")
    table, wf = CF.build_transfer(m.weight, m.bias, 1, 1e-5, 268, 268)
    x = torch.randn(2, 64, 256, 256, device="cuda")
    with torch.no_grad():
        assert torch.equal(CF.converse2d_forward(x, table, wf, 3, 1, 6, "circular"), m(x))


def test_training_at_268_reads_one_table():
    """Full pairs of planes of 268 x 268, 128 of them or more: the integer contractions with and without gradients, and of
    the two tables the one that they and the backward read; fewer planes: the pair kernels and both tables."""
    from conversenet_b200 import Converse2D, ConverseBlock, _cabi
    torch.manual_seed(5)
    bytes_of = lambda C: _cabi.load().cvb_plane_transfer_bytes(C, 268, 268)
    x = torch.randn(2, 64, 256, 256, device="cuda")
    for C, alone in ((64, True), (8, False)):
        m = Converse2D(C, C, 7, padding=6, padding_mode="circular").cuda()
        y = m(x[:, :C])
        assert ({t.numel() for t, _ in m._tables.values()} == {bytes_of(C)}) == alone
        m.weight.requires_grad_(False), m.bias.requires_grad_(False)
        z = m(x[:, :C].clone().requires_grad_(True))
        with torch.no_grad():
            assert torch.equal(m(x[:, :C]), y) and torch.equal(z, y)
    blk = ConverseBlock(64, 64, 7, 1, 6, "circular").cuda()
    y = blk(x)
    assert {t.numel() for t, _ in blk.conv1[3]._tables.values()} == {bytes_of(128)}
    with torch.no_grad():
        assert _rel(blk(x), y) <= 1e-6


def test_integer_contractions_keep_planes_apart():
    from conversenet_b200 import Converse2D
    g = torch.Generator(device="cuda").manual_seed(3)
    m = Converse2D(96, 96, 3, padding=1, padding_mode="circular").cuda().eval()
    x = torch.randn(1, 96, 242, 266, device="cuda", generator=g)
    with torch.no_grad():
        y = m(x)
        z = x.clone()
        z[0, 7, 100, 3], z[0, 50, 0, 0] = float("nan"), float("inf")
        z[0, 20] *= 2.0 ** 60
        t = m(z)
    same = [c for c in range(96) if c not in (7, 20, 50)]
    assert torch.equal(t[:, same], y[:, same]) and torch.equal(t[:, 20], y[:, 20] * 2.0 ** 60)
    assert bool(t[0, 7].isnan().all()) and not bool(t[0, 50].isfinite().any())


@pytest.mark.parametrize("case", [
    # lengths above 680: dense stages of 64, 80, 60 and 95 points (real planes), two register radices (832 = 32 * 26)
    (2, 1, 1022, 130, 3, 1, 1, "circular", "fp32"),
    (1, 2, 60, 1278, 5, 1, 1, "replicate", "bf16"),
    (2, 1, 896, 77, 3, 2, 2, "reflect", "fp32"),
    (1, 1, 1043, 828, 3, 1, 2, "constant", "fp32"),       # 1047 = 3 * 349 is refused
    (1, 1, 1040, 828, 3, 1, 2, "constant", "fp32"),       # 1044 = 87 * 12
    (1, 1, 1300, 805, 3, 1, 0, "circular", "fp32"),       # the longest dense axis; alone in its batch
    # both lengths with a costly dense stage: full pairs take the three-stage plans of the pair kernels
    (2, 1, 803, 889, 3, 1, 1, "circular", "fp32"),
    (7, 1, 914, 914, 7, 1, 2, "reflect", "bf16"),         # an odd batch: the last pair holds one plane
    (2, 1, 874, 1249, 3, 1, 0, "replicate", "fp32"),      # 874 has the prime 23, 1249 is prime: refused
    (2, 1, 873, 1248, 3, 1, 1, "constant", "fp32"),       # 875 = 7 * 5 * 5 * 5, 1250: four stages
    (4, 1, 803, 889, 3, 2, 1, "circular", "fp32"),        # scale 2: real planes
])
def test_long_axes_match_the_oracle(case):
    from conversenet_b200 import Converse2D
    B, C, H, W, k, s, p, mode, dt = case
    rng = np.random.default_rng(H + W)
    w, b = orc.init_weight(C, k, rng)
    dtype = torch.float32 if dt == "fp32" else torch.bfloat16
    x = torch.from_numpy(rng.standard_normal((B, C, H, W)).astype(np.float32)).to(dtype)
    m = Converse2D(C, C, k, scale=s, padding=p, padding_mode=mode).cuda().eval()
    with torch.no_grad():
        m.weight.copy_(torch.from_numpy(w))
        m.bias.copy_(torch.from_numpy(b))
        if H + 2 * p == 1047 or W + 2 * p == 1249:
            with pytest.raises(RuntimeError):
                m(x.cuda())
            return
        y = m(x.cuda()).float().cpu().numpy()
        m.fuse_gelu = True
        gelu = m(x.cuda()).float().cpu()
    ref = orc.converse2d_forward(x.float().numpy(), w, b, s, p, mode, 1e-5, dtype=np.float64)
    assert orc.rel_l2(y, ref) <= (2e-6 if dt == "fp32" else 3e-3)
    want = torch.nn.functional.gelu(torch.from_numpy(ref)).numpy()
    assert orc.rel_l2(gelu.numpy(), want) <= (4e-6 if dt == "fp32" else 3e-3)


@pytest.mark.parametrize("n,planes,s", [
    (76, 2, 2), (108, 98, 1), (108, 99, 2),          # below 96 KB of shared memory: one block at any count
    (110, 98, 1), (110, 99, 1), (132, 99, 2),        # above: from two thirds of the SMs on
    (96, 148, 1), (96, 149, 1), (110, 149, 2),       # one plane more than SMs
    (136, 148, 1),                                   # the largest that one block takes
])
def test_one_block_per_plane_and_three_launches_agree(n, planes, s):
    """Both sides of the lines between the two forms (148 SMs), and the same call forced through the launches."""
    from conversenet_b200 import Converse2D, _cabi
    torch.manual_seed(n + planes)
    m = Converse2D(planes, planes, 5, scale=s, padding=2).cuda().eval()
    x = torch.randn(1, planes, n - 4, n - 4, device="cuda")
    with torch.no_grad():
        y = m(x)
        with _cabi.option(_cabi.OPT_MULTIPASS, 1):
            z = m(x)
    assert _rel(y, z) <= 1e-6
    c = planes // 2
    ref = orc.converse2d_forward(x[:, c:c + 1].cpu().numpy(), m.weight[:, c:c + 1].detach().cpu().numpy(),
                                 m.bias[:, c:c + 1].detach().cpu().numpy(), s, 2, "circular", 1e-5, dtype=np.float64)
    assert orc.rel_l2(y[:, c:c + 1].cpu().numpy(), ref) <= 2e-6


def test_chunks_of_the_workspace_agree_with_single_planes():
    # 320 planes of 300 x 260 need several chunks; one plane alone needs one
    from conversenet_b200 import Converse2D
    torch.manual_seed(1)
    m = Converse2D(160, 160, 3, padding=0).cuda().eval()
    x = torch.randn(2, 160, 300, 260, device="cuda")
    with torch.no_grad():
        y = m(x)
        one = Converse2D(1, 1, 3, padding=0).cuda().eval()
        for c in (0, 77, 159):
            one.weight.copy_(m.weight[:, c:c + 1])
            one.bias.copy_(m.bias[:, c:c + 1])
            assert _rel(y[1:, c:c + 1], one(x[1:, c:c + 1].contiguous())) <= 1e-6


@pytest.mark.parametrize("case", [
    (2, 3, 24, 31, 3, 1, 3, "replicate"),
    (3, 2, 33, 41, 5, 1, 2, "reflect"),        # 37 x 45: dense stage along y
    (2, 2, 30, 49, 3, 2, 2, "circular"),       # 34 x 53: dense stage along x
    (1, 2, 60, 63, 7, 1, 2, "constant"),       # 64 x 67
    (2, 2, 16, 18, 5, 3, 2, "circular"),       # odd scale
    (2, 2, 15, 14, 4, 4, 1, "replicate"),      # run-time taps and scale
    (2, 3, 15, 18, 7, 3, 3, "reflect"),        # the largest window of a compile-time adjoint epilogue at an odd scale
    (4, 3, 64, 64, 5, 2, 2, "reflect"),        # r kept by the pair kernels
    (2, 2, 12, 12, 3, 5, 1, "circular"),       # scale without native parameter gradients
    (2, 2, 12, 9, 3, 1, 8, "circular"),        # margins almost as wide as the plane
])
def test_gradients_match_fp64_autograd(case):
    from conversenet_b200 import Converse2D
    from conversenet_b200.autograd import spectral_forward
    B, C, H, W, k, s, p, mode = case
    torch.manual_seed(H + W)
    m = Converse2D(C, C, k, scale=s, padding=p, padding_mode=mode).cuda()
    with torch.no_grad():
        m.bias.add_(torch.randn_like(m.bias) + 4.0)
    x = torch.randn(B, C, H, W, device="cuda", requires_grad=True)
    y = m(x)
    g = torch.randn_like(y)
    got = torch.autograd.grad(y, (x, m.weight, m.bias), g)
    a = [t.detach().double().requires_grad_(True) for t in (x, m.weight, m.bias)]
    ref = torch.autograd.grad(spectral_forward(*a, s, p, mode, 1e-5), a, g.double())
    for q, r in zip(got, ref):
        assert _rel(q, r) <= 2e-5


@pytest.mark.parametrize("params", [False, True])       # dL/dx alone sends the rows through the contractions as well
@pytest.mark.parametrize("case", [
    (1, 96, 132, 140, 3, 1, 1, "circular"),    # 134 x 142
    (2, 24, 250, 232, 3, 1, 4, "reflect"),     # 258 x 240: columns alone
    (1, 64, 256, 256, 7, 1, 6, "replicate"),   # 268 x 268
    (1, 96, 242, 131, 3, 2, 1, "constant"),    # 244 x 133 by 2
    (1, 3, 200, 192, 5, 1, 1, "circular"),     # 202 x 194: wide dense stages, any number of planes
])
def test_gradients_through_the_integer_contractions(case, params):
    from conversenet_b200 import Converse2D, _cabi
    from conversenet_b200.autograd import spectral_forward
    B, C, H, W, k, s, p, mode = case
    torch.manual_seed(H + W)
    m = Converse2D(C, C, k, scale=s, padding=p, padding_mode=mode).cuda()
    with torch.no_grad():
        m.bias.add_(torch.randn_like(m.bias) + 4.0)
    m.requires_grad_(params)
    x = torch.randn(B, C, H, W, device="cuda", requires_grad=True)
    of = [x, m.weight, m.bias] if params else [x]
    y = m(x)
    g = torch.randn_like(y)
    got = torch.autograd.grad(y, of, g)
    a = [t.detach().double().requires_grad_(True) for t in (x, m.weight, m.bias)]
    ref = torch.autograd.grad(spectral_forward(*a, s, p, mode, 1e-5), a[:len(of)], g.double())
    assert _rel(got[0], ref[0]) <= 6e-7          # tests/test_emu_rp.py
    for q, r in zip(got[1:], ref[1:]):
        assert _rel(q, r) <= 2e-6                # sums over every pixel, the chain rule in 64 bits
    assert _cabi.load().cvb_last_device_status(1) == 0


@pytest.mark.parametrize("case", [
    (1, 2, 20, 130, 5, 2, 2, "circular"),      # 67 items side by side: two tiles
    (1, 1, 61, 36, 3, 2, 1, "replicate"),      # odd rows and columns of items, several tiles down, 16-byte copies
    (2, 1, 19, 27, 7, 2, 0, "circular"),       # the windows wrap around; 4-byte copies
    (1, 1, 18, 20, 7, 2, 0, "reflect"),        # the windows wrap around; 16-byte copies
    (1, 1, 9, 138, 7, 4, 3, "constant"),       # the widest tiles
    (1, 2, 12, 44, 3, 3, 4, "replicate"),      # odd scale, 16-byte copies
    (1, 1, 2, 2, 2, 2, 0, "circular"),
])
def test_upsampling_gradients_across_tiles(case):
    # the bound of test_gradients_match_fp64_autograd: the fp32 transforms' error, which the tiles leave as it is
    test_gradients_match_fp64_autograd(case)


@pytest.mark.parametrize("B,H,W", [(1, 4, 5), (3, 24, 31), (2, 16, 16), (1, 37, 64)])
@pytest.mark.parametrize("alphas", [False, True])
def test_block_and_its_gradients_match_the_layer_by_layer_block(monkeypatch, B, H, W, alphas):
    """Pixel counts that are no multiple of a 128-pixel tile, of a 32-pixel tile, fewer than one tile."""
    from conversenet_b200 import ConverseBlock, ConverseBlockAlphaVariant
    from conversenet_b200 import util_converse as uc
    monkeypatch.setattr(torch.backends.cudnn, "allow_tf32", False)      # the library convolutions' gradients
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", False)
    torch.manual_seed(H)
    blk = (ConverseBlockAlphaVariant if alphas else ConverseBlock)(64, 64, 3, 1, 2, "circular").cuda()
    with torch.no_grad():
        for q in blk.parameters():
            if q.dim() == 1 or q.shape[-1] == 1 and q.shape[0] == 1:
                q.add_(0.2 * torch.randn_like(q))
    x = torch.randn(B, 64, H, W, device="cuda", requires_grad=True)
    g = torch.randn_like(x)

    def step():
        y = blk(x)
        return [y] + list(torch.autograd.grad(y, [x] + list(blk.parameters()), g))

    with torch.no_grad():
        inference = blk(x)
    fused = step()
    monkeypatch.setattr(uc, "BLOCK_FUSION", False)
    plain = step()
    assert _rel(inference, plain[0]) <= 2e-6
    for a, r in zip(fused, plain):
        assert float((a - r).norm()) <= 2e-5 * float(r.norm()) + 1e-6
    from conversenet_b200 import _cabi
    assert _cabi.load().cvb_last_device_status(1) == 0


def _block_fp64(q, conv, mode, x):
    """ConverseBlock in 64 bits: q the fourteen parameters of functional.block_parameters (None for absent alphas)."""
    from conversenet_b200.autograd import spectral_forward
    F = torch.nn.functional

    def norm(v, w, b):
        u = v.mean(1, keepdim=True)
        return (v - u) / torch.sqrt((v - u).pow(2).mean(1, keepdim=True) + 1e-5) * w[:, None, None] + b[:, None, None]
    t = F.gelu(F.conv2d(norm(x, q[0], q[1]), q[2], q[3]))
    t = F.gelu(spectral_forward(t, conv[0], conv[1], 1, conv[2], mode, 1e-5))
    x1 = x + (1.0 if q[6] is None else q[6]) * F.conv2d(t, q[4], q[5])
    return x1 + (1.0 if q[13] is None else q[13]) * F.conv2d(F.gelu(F.conv2d(norm(x1, q[7], q[8]), q[9], q[10])), q[11], q[12])


@pytest.mark.parametrize("B,H,W", [(1, 4, 5), (2, 64, 64), (5, 33, 47)])
def test_block_gradients_match_fp64(B, H, W):
    """Every gradient of a block against 64 bits: less than one tile of 32 pixels, one or two a block of the weight
    gradients, several with a short last one."""
    from conversenet_b200 import ConverseBlockAlphaVariant
    from conversenet_b200 import _cabi, functional as CF
    torch.manual_seed(H)
    blk = ConverseBlockAlphaVariant(64, 64, 5, 1, 4, "replicate").cuda()
    with torch.no_grad():
        for q in blk.parameters():
            if q.dim() == 1 or q.shape[-1] == 1 and q.shape[0] == 1:
                q.add_(0.2 * torch.randn_like(q))
    c1, c2 = blk.conv1, blk.conv2
    params = list(CF.block_parameters(c1[0], c1[1], c1[5], blk.alpha1, c2[0], c2[1], c2[3], blk.alpha2)) + [c1[3].weight, c1[3].bias]
    x = torch.randn(B, 64, H, W, device="cuda", requires_grad=True)
    y = blk(x)
    g = torch.randn_like(y)
    got = [y] + list(torch.autograd.grad(y, [x] + params, g))
    a = [t.detach().double().requires_grad_(True) for t in [x] + params]
    ref = _block_fp64(a[1:15], (a[15], a[16], 4), "replicate", a[0])
    want = [ref] + list(torch.autograd.grad(ref, a, g.double()))
    assert _cabi.load().cvb_last_device_status(1) == 0
    # TF32 hi + lo is within 2^-22 of a value and lo lo (2^-24) is left out: below the rounding of fp32 sums of as many
    # pixels; a bit of the operands lost would be 1e-5
    errors = [_rel(u, v) for u, v in zip(got, want)]
    assert max(errors) <= 2e-6, errors


@pytest.mark.parametrize("B,H,W", [(3, 41, 64), (5, 33, 47)])
def test_block_gradients_over_several_tiles_of_pixels(monkeypatch, B, H, W):
    """246 and 243 tiles of 32 pixels: three or four a block of the weight gradients, so that both operand buffers are reused."""
    test_block_and_its_gradients_match_the_layer_by_layer_block(monkeypatch, B, H, W, True)


def test_block_follows_its_parameters():
    from conversenet_b200 import ConverseBlock
    torch.manual_seed(3)
    blk = ConverseBlock(64, 64, 3, 1, 2, "circular").cuda().eval()
    x = torch.randn(1, 64, 24, 20, device="cuda")
    with torch.no_grad():
        a = blk(x)
        blk.conv2[3].bias.add_(1.0)
        b = blk(x)
    assert _rel(b - a, torch.ones_like(a)) <= 1e-5


def test_bf16_network_keeps_the_pair_kernels():
    from conversenet_b200 import functional as CF
    from conversenet_b200.models import ConverseDnCNN
    torch.manual_seed(4)
    net = ConverseDnCNN().cuda().eval()
    net.activation_dtype = torch.bfloat16
    assert all(b.fixed_order for b in net.m_body)
    blk = net.m_body[0]
    conv = blk.conv1[3]
    x = torch.randn(3, 64, 40, 37, device="cuda").bfloat16()       # 52 x 49, an unpaired plane
    with torch.no_grad():
        y = blk(x)
        t = CF.ln_pw_gelu(x, blk.conv1[0], blk.conv1[1])
        table, wf = CF.build_pair_transfer(conv.weight, conv.bias, conv.eps, 52, 49)
        u = CF.pair_forward(t, table, wf, 7, 6, "circular", fuse_gelu=True)
        z = CF.pw_res_mlp(u, x, blk.conv1[5], blk.conv2[0], blk.conv2[1], blk.conv2[3])
    assert torch.equal(y, z)
    conv.fuse_gelu = True
    with torch.no_grad():
        ref = conv(t.float())
    conv.fuse_gelu = False
    assert _rel(u, ref) <= 3e-3
    net.activation_dtype = None
    assert not any(b.fixed_order for b in net.m_body)
