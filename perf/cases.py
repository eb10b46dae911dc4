"""Performance cases: what programs that use this package have it do, through its public entry points.

Five kinds of pass, each over a range of sizes:

  layer        one Converse2D forward without gradients (fp32 or bf16 tensors, scale 1 to 4)
  block        one ConverseBlock forward without gradients (64 channels, the settings of the three networks)
  net          one forward of ConverseDnCNN, ConverseMSRResNet or ConverseUSRNet, eager or replayed from a CUDA graph
  train_layer  one training step of a Converse2D layer: forward, all gradients, SGD update
  train_block  the same for a ConverseBlock

`listed()` holds one or a few named cases of each kind, `draw(rng)` more of the same ranges.
"""
import math

import torch

from conversenet_b200 import Converse2D, ConverseBlock, ConverseBlockAlphaVariant
from conversenet_b200.graphs import GraphedForward
from conversenet_b200.models import ConverseDnCNN, ConverseMSRResNet, ConverseUSRNet

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
MODES = ("circular", "replicate", "reflect", "constant")

# (kernel size, padding, padding mode, per-channel branch scales) of the blocks of the three networks
BLOCKS = {
    "dncnn": (7, 6, "circular", False),
    "srresnet": (5, 4, "replicate", False),
    "usrnet": (3, 2, "circular", True),
}


def _layer(name, B, C, H, W, k, s, p, mode, dtype):
    return {"name": name, "kind": "layer", "B": B, "C": C, "H": H, "W": W, "k": k, "s": s, "p": p, "mode": mode,
            "dtype": dtype}


def listed():
    return [
        # The smallest call: one small tile or feature map through one layer. Latency and launches.
        _layer("layer_small", 1, 64, 24, 20, 3, 1, 2, "replicate", "fp32"),
        # One image through one layer (benchmark configuration 1).
        _layer("layer_image", 1, 64, 128, 128, 5, 1, 2, "circular", "fp32"),
        # The upsampling layer on a batch (benchmark configuration 2), fp32.
        _layer("layer_up2", 16, 64, 64, 64, 5, 2, 2, "circular", "fp32"),
        # A ragged feature map upsampled by 3 on bf16 tensors.
        _layer("layer_up3_ragged_bf16", 4, 48, 77, 118, 3, 3, 1, "reflect", "bf16"),
        # A whole photograph (a 321 x 481 picture) through a denoiser's 128-channel layer, unpadded to any round size.
        _layer("layer_photo", 1, 128, 321, 481, 7, 1, 6, "circular", "fp32"),
        # The denoiser's block at the benchmark's batch and resolution (configuration 3).
        {"name": "block_dncnn", "kind": "block", "block": "dncnn", "B": 8, "H": 256, "W": 256, "dtype": "fp32"},
        # The super-resolution block on bf16 tensors of an odd size.
        {"name": "block_srresnet_odd_bf16", "kind": "block", "block": "srresnet", "B": 2, "H": 111, "W": 167,
         "dtype": "bf16"},
        # Denoising one picture, eager.
        {"name": "net_dncnn", "kind": "net", "net": "dncnn", "B": 1, "H": 256, "W": 256, "sf": 1, "graph": False,
         "dtype": "fp32"},
        # Super-resolution x4 of a batch, served from a CUDA graph (configuration 4 at a quarter of its batch).
        {"name": "net_srresnet_graph", "kind": "net", "net": "srresnet", "B": 4, "H": 128, "W": 128, "sf": 4,
         "graph": True, "dtype": "fp32"},
        # Non-blind deblurring and super-resolution x2 of one picture of an ordinary, not round size, eager.
        {"name": "net_usrnet", "kind": "net", "net": "usrnet", "B": 1, "H": 120, "W": 160, "sf": 2, "graph": False,
         "dtype": "fp32"},
        # Training steps on patches.
        {"name": "train_layer_up2", "kind": "train_layer", "B": 16, "C": 64, "H": 64, "W": 64, "k": 5, "s": 2, "p": 2,
         "mode": "circular"},
        {"name": "train_block_dncnn", "kind": "train_block", "block": "dncnn", "B": 8, "H": 64, "W": 64},
    ]


# ------------------------------------------------------------------ drawn cases
def _supported(n):
    """Padded lengths the operator accepts: at least 2, no prime factor above 127."""
    if n < 2:
        return False
    f = 2
    while f * f <= n:
        while n % f == 0:
            n //= f
        f += 1
    return n <= 127


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _padded(case):
    """Every padded length a case transforms."""
    kind = case["kind"]
    out = []
    for n in (case["H"], case["W"]):
        if kind in ("layer", "train_layer"):
            out.append(n + 2 * case["p"])
        elif kind in ("block", "train_block"):
            out.append(n + 2 * BLOCKS[case["block"]][1])
        elif case["net"] == "dncnn":
            out.append(n + 12)
        elif case["net"] == "srresnet":
            out += [n + 8, n + 4, 2 * n + 8, 2 * n + 4, 4 * n + 8]
        else:
            out += [n, n * case["sf"], n * case["sf"] + 4]
    return out


def _draw_once(rng):
    kind = rng.choice(["layer"] * 5 + ["block"] * 2 + ["net"] * 3 + ["train_layer"] + ["train_block"])
    if kind in ("layer", "train_layer"):
        train = kind == "train_layer"
        s = rng.choice([1, 1, 2, 2] if train else [1, 1, 1, 2, 2, 3, 4])
        k = rng.choice([3, 5, 7] + ([2] if s == 2 else []))
        case = {"kind": kind, "B": _log_int(rng, 2, 16) if train else _log_int(rng, 1, 16),
                "C": _log_int(rng, 16, 128), "k": k, "s": s, "p": rng.randint(k // 2, max(k // 2, k - 1)),
                "mode": rng.choice(MODES)}
        lo, hi = (24, 130) if train else (16, 520)
        case["H"] = _log_int(rng, lo, hi)
        case["W"] = min(hi, max(lo, int(case["H"] * rng.uniform(0.6, 1.7))))
        pixels = case["B"] * case["C"] * case["H"] * case["W"] * s * s
        if pixels > (16 * 64 * 128 * 128 if train else 8 * 64 * 256 * 256):
            return None
        if not train:
            case["dtype"] = rng.choice(["fp32", "fp32", "bf16"])
        return case
    if kind in ("block", "train_block"):
        train = kind == "train_block"
        lo, hi = (24, 130) if train else (24, 300)
        case = {"kind": kind, "block": rng.choice(sorted(BLOCKS)), "B": _log_int(rng, 2 if train else 1, 8),
                "H": _log_int(rng, lo, hi)}
        case["W"] = min(hi, max(lo, int(case["H"] * rng.uniform(0.6, 1.7))))
        if rng.random() < 0.4:      # networks also run on whole tiles
            case["H"], case["W"] = max(32, case["H"] // 32 * 32), max(32, case["W"] // 32 * 32)
        if case["B"] * case["H"] * case["W"] > (8 * 64 * 64 if train else 8 * 256 * 256):
            return None
        if not train:
            case["dtype"] = rng.choice(["fp32", "fp32", "bf16"])
        return case
    net = rng.choice(["dncnn", "srresnet", "usrnet"])
    sf = {"dncnn": 1, "srresnet": 4, "usrnet": rng.randint(1, 4)}[net]
    case = {"kind": "net", "net": net, "B": rng.choice([1, 1, 2, 4]), "sf": sf, "graph": rng.random() < 0.4,
            "dtype": rng.choice(["fp32", "fp32", "bf16"]) if net == "dncnn" else "fp32"}
    lo, hi = {"dncnn": (48, 300), "srresnet": (24, 130), "usrnet": (48, 330)}[net]
    case["H"] = _log_int(rng, lo, hi)
    case["W"] = min(hi, max(lo, int(case["H"] * rng.uniform(0.6, 1.7))))
    if rng.random() < 0.5:
        case["H"], case["W"] = max(32, case["H"] // 32 * 32), max(32, case["W"] // 32 * 32)
    most = {"dncnn": 256 * 256, "srresnet": 4 * 128 * 128, "usrnet": 320 * 320 / (sf * sf)}[net]
    return case if case["B"] * case["H"] * case["W"] <= most else None


def draw(rng):
    while True:
        case = _draw_once(rng)
        if case is not None and all(_supported(n) for n in _padded(case)):
            return case


# ------------------------------------------------------------------ one case
def _exact_library_convolutions():
    # fp32 programs that care about their results run the networks' 1x1 head and tail without TF32
    torch.backends.cudnn.allow_tf32 = False
    torch.backends.cuda.matmul.allow_tf32 = False


def _seeded(make, seed):
    """A module with its own initialisation, drawn from `seed`, on the GPU."""
    with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
        torch.manual_seed(seed)
        return make().cuda()


def _jitter(module, g):
    """Parameters as training leaves them: biases, branch scales and norms off their initial constants."""
    with torch.no_grad():
        for n, q in module.named_parameters():
            r = torch.randn(q.shape, device=q.device, generator=g)
            if n.endswith(("alpha1", "alpha2")):
                q.copy_(0.1 * r)
            elif n.endswith("d.alpha"):
                q.copy_(9.0 + r)
            elif q.dim() == 4 and q.shape[0] == 1 and q.shape[-1] == 1:    # Converse2D bias
                q.copy_(0.5 * r)
            elif q.dim() == 1:
                q.add_(0.05 * r)


def _smooth_images(B, c, H, W, g):
    """Images in [0, 1]: smooth fields, as photographs mostly are."""
    x = torch.randn(B, c, H + 16, W + 16, device="cuda", generator=g)
    for _ in range(2):
        x = torch.nn.functional.avg_pool2d(x, 9, stride=1)
    x = x - x.amin(dim=(1, 2, 3), keepdim=True)
    return (x / x.amax(dim=(1, 2, 3), keepdim=True)).contiguous()


def _blur_kernels(B, g):
    """Anisotropic Gaussian 7 x 7 blur kernels (widths 0.6 to 3 px, any rotation), normalised."""
    u = torch.rand(B, 3, device="cuda", generator=g)
    sx, sy, th = 0.6 + 2.4 * u[:, 0], 0.6 + 2.4 * u[:, 1], math.pi * u[:, 2]
    r = torch.arange(7, device="cuda", dtype=torch.float32) - 3
    yy, xx = r[:, None], r[None, :]
    c, s = torch.cos(th).view(B, 1, 1), torch.sin(th).view(B, 1, 1)
    a, b = (c * xx + s * yy) / sx.view(B, 1, 1), (c * yy - s * xx) / sy.view(B, 1, 1)
    k = torch.exp(-0.5 * (a * a + b * b))
    return (k / k.sum(dim=(1, 2), keepdim=True)).unsqueeze(1).contiguous()


def _block_module(block):
    k, p, mode, alphas = BLOCKS[block]
    return (ConverseBlockAlphaVariant if alphas else ConverseBlock)(64, 64, k, 1, p, mode)


def prepare(case, seed):
    _exact_library_convolutions()
    kind = case["kind"]
    B, H, W = case["B"], case["H"], case["W"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("layer", "train_layer"):
        C, s = case["C"], case["s"]
        m = _seeded(lambda: Converse2D(C, C, case["k"], scale=s, padding=case["p"], padding_mode=case["mode"]), seed)
        shape, out_shape = (B, C, H, W), (B, C, H * s, W * s)
    elif kind in ("block", "train_block"):
        m = _seeded(lambda: _block_module(case["block"]), seed)
        shape = out_shape = (B, 64, H, W)
    else:
        m = _seeded({"dncnn": ConverseDnCNN, "srresnet": ConverseMSRResNet, "usrnet": ConverseUSRNet}[case["net"]], seed)
    _jitter(m, g)

    if kind == "net":
        m.eval()
        args = [_smooth_images(B, 1 if case["net"] == "dncnn" else 3, H, W, g)]
        if case["net"] == "dncnn":
            args[0] += 25.0 / 255.0 * torch.randn(args[0].shape, device="cuda", generator=g)
            if case["dtype"] == "bf16":
                m.activation_dtype = torch.bfloat16
        elif case["net"] == "usrnet":
            args += [_blur_kernels(B, g), case["sf"]]
        return {"kind": kind, "call": GraphedForward(m, *args) if case["graph"] else m, "args": args}

    x = torch.randn(shape, device="cuda", generator=g)
    if kind in ("layer", "block"):
        m.eval()
        return {"kind": kind, "call": m, "args": [x.to(DTYPES[case["dtype"]])]}

    # training: the layer's input comes from earlier layers (it needs a gradient too), and the gradient of a mean
    # loss comes back from later ones
    n = math.prod(out_shape)
    return {"kind": kind, "call": m, "x": x.requires_grad_(True), "params": list(m.parameters()),
            "grad_out": torch.randn(out_shape, device="cuda", generator=g) / n,
            "optimizer": torch.optim.SGD(m.parameters(), lr=1e-4)}


def run(state):
    if state["kind"] in ("layer", "block", "net"):
        with torch.no_grad():
            return state["call"](*state["args"])
    x, opt = state["x"], state["optimizer"]
    opt.zero_grad(set_to_none=True)
    x.grad = None
    y = state["call"](x)
    y.backward(state["grad_out"])
    opt.step()
    return {"y": y.detach(), "dx": x.grad, "dparams": [q.grad for q in state["params"]],
            "params": [q.detach() for q in state["params"]]}


# ------------------------------------------------------------------ what a pass cannot do without
def _solve_flops(planes, H, W, k, s, p):
    """Two real FFTs of every padded plane, the multiply, and the k x k correlation of the upsampling form."""
    n = (H + 2 * p) * (W + 2 * p)
    f = 2 * 2.5 * n * math.log2(n) + 3 * n
    if s > 1:
        f += 2.0 * k * k * H * W + s * s * H * W
    return planes * f


def _block_flops(block, B, H, W):
    k, p, _, _ = BLOCKS[block]
    return B * H * W * 4 * 2 * 64 * 128 + _solve_flops(B * 128, H, W, k, 1, p)


def work(case):
    kind, B, H, W = case["kind"], case["B"], case["H"], case["W"]
    e = 2 if case.get("dtype") == "bf16" else 4
    if kind in ("layer", "train_layer"):
        C, k, s = case["C"], case["k"], case["s"]
        n_in = B * C * H * W
        flops = _solve_flops(B * C, H, W, k, s, case["p"])
        weights = C * (k * k + 1)
        if kind == "layer":
            return {"bytes": e * n_in * (1 + s * s) + 4 * weights, "flops": flops}
        # x and dL/dy in, y and dL/dx out, parameters in and out with their gradients; three transform pairs
        return {"bytes": 4 * (2 * n_in * (1 + s * s) + 3 * weights), "flops": 3 * flops}
    if kind in ("block", "train_block"):
        n, flops = B * 64 * H * W, _block_flops(case["block"], B, H, W)
        weights = 4 * 64 * 128 + 128 * BLOCKS[case["block"]][0] ** 2 + 900
        if kind == "block":
            return {"bytes": 2 * e * n + 4 * weights, "flops": flops}
        return {"bytes": 4 * (4 * n + 3 * weights), "flops": 3 * flops}
    net, sf = case["net"], case["sf"]
    if net == "dncnn":
        flops, weights, io = 20 * _block_flops("dncnn", B, H, W), 796353, 2 * B * H * W
    elif net == "srresnet":
        flops = (17 * _block_flops("srresnet", B, H, W) + _block_flops("srresnet", B, 2 * H, 2 * W)
                 + _block_flops("srresnet", B, 4 * H, 4 * W)
                 + _solve_flops(B * 64, H, W, 2, 2, 2) + _solve_flops(B * 64, 2 * H, 2 * W, 2, 2, 2))
        weights, io = 699072, 3 * B * H * W * 17
    else:
        Hs, Ws = H * sf, W * sf
        flops = (35 * _block_flops("usrnet", B, Hs, Ws) + _solve_flops(B * 64, H, W, 7, sf, 0)
                 + 4 * _solve_flops(B * 64, Hs, Ws, 7, 1, 0))
        weights, io = 307987, 3 * B * (H * W + Hs * Ws)
    return {"bytes": 4 * (io + weights), "flops": flops}


def tolerance(case):
    """fp32: the rounding of sums of a few hundred 32-bit values; a network of random weights amplifies it block after
    block (measured against fp64: up to 1e-4).  bf16 tensors round every value to 8 bits of mantissa, a block or a
    network several times."""
    kind = case["kind"]
    if case.get("dtype") == "bf16":
        return {"rel": 4e-3 if kind == "layer" else 1e-2, "max": 0.1}
    return {"rel": {"layer": 1e-5, "block": 2e-5, "net": 4e-4, "train_layer": 5e-5, "train_block": 5e-5}[kind],
            "max": 5e-3}
