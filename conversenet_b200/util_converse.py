"""Drop-in for the reference's `models/util_converse.py`: same class names, constructor
signatures, parameter names/shapes and forward semantics; the arithmetic runs in
hand-written sm_100a kernels behind the C ABI, under autograd too (`autograd.py`)."""
import os
from collections import OrderedDict

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import _cabi, functional as CF
from ._kept import Kept
from .autograd import Converse2DFunction, ConverseBlockFunction


# False: ConverseBlock runs its layers one by one (PyTorch LayerNorm / 1x1 / GELU around the native
# operator) instead of the fused block kernels; the tests compare the two.
BLOCK_FUSION = True


class _exact_fp32:
    """PyTorch's 1x1 convolutions (cuDNN / cuBLAS) in full fp32 for a block of code.  The unfused route of
    ConverseBlock (channel counts other than 64, or autograd) must hold the operator's 1e-4 bar, which
    TF32 (10-bit mantissa, on by default for cuDNN convolutions) does not."""

    def __enter__(self):
        self.saved = (torch.backends.cudnn.allow_tf32, torch.backends.cuda.matmul.allow_tf32)
        torch.backends.cudnn.allow_tf32 = False
        torch.backends.cuda.matmul.allow_tf32 = False

    def __exit__(self, *exc):
        torch.backends.cudnn.allow_tf32, torch.backends.cuda.matmul.allow_tf32 = self.saved
        return False


class LayerNorm(nn.Module):
    """channels_last / channels_first LayerNorm (`models/util_converse.py:42-68`)."""

    def __init__(self, normalized_shape, eps=1e-6, data_format="channels_last"):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(normalized_shape))
        self.bias = nn.Parameter(torch.zeros(normalized_shape))
        self.eps = eps
        self.data_format = data_format
        if self.data_format not in ["channels_last", "channels_first"]:
            raise NotImplementedError
        self.normalized_shape = (normalized_shape,)

    def forward(self, x):
        if self.data_format == "channels_last":
            return F.layer_norm(x, self.normalized_shape, self.weight, self.bias, self.eps)
        u = x.mean(1, keepdim=True)
        s = (x - u).pow(2).mean(1, keepdim=True)
        x = (x - u) / torch.sqrt(s + self.eps)
        return self.weight[:, None, None] * x + self.bias[:, None, None]


def sequential(*args):
    """Flattening `nn.Sequential` builder (`models/util_converse.py:71-91`)."""
    if len(args) == 1:
        if isinstance(args[0], OrderedDict):
            raise NotImplementedError("sequential does not support OrderedDict input.")
        return args[0]
    modules = []
    for module in args:
        if isinstance(module, nn.Sequential):
            modules.extend(module.children())
        elif isinstance(module, nn.Module):
            modules.append(module)
    return nn.Sequential(*modules)


class Converse2D(nn.Module):
    """Depthwise reverse convolution (`models/util_converse.py:98-192`).

    `Converse2D(in_channels, out_channels, kernel_size, scale=1, padding=2,
    padding_mode='circular', eps=1e-5, backend='auto')`, parameters
    `weight (1,C,k,k)` (softmax-normalised normal draw) and `bias (1,C,1,1)`
    (zeros), `forward(x: (B,C,H,W)) -> (B,C,H*scale,W*scale)`.

    With autograd enabled and an input or parameter that requires a gradient the call is
    differentiable (`conversenet_b200/autograd.py`: dL/dx through the native kernels).

    `backend` is accepted for compatibility: 'auto' and 'cuda' run the native
    kernels; 'pytorch' (or CONVERSE2D_BACKEND=pytorch) raises, because this build
    carries no torch.fft path.  The output is contiguous (the reference returns a
    cropped view)."""

    _TABLE_SLOTS = 8

    def __init__(self, in_channels, out_channels, kernel_size, scale=1, padding=2, padding_mode="circular",
                 eps=1e-5, backend="auto"):
        super().__init__()
        self.in_channels = in_channels
        self.out_channels = out_channels
        self.kernel_size = kernel_size
        self.scale = scale
        self.padding = padding
        self.padding_mode = padding_mode
        self.eps = eps
        self.backend = backend.lower()
        if self.backend not in ("auto", "cuda", "pytorch"):
            raise ValueError(f"backend must be 'auto' | 'cuda' | 'pytorch', got: {self.backend}")
        assert self.out_channels == self.in_channels  # depthwise
        self.weight = nn.Parameter(torch.randn(1, self.in_channels, self.kernel_size, self.kernel_size))
        self.bias = nn.Parameter(torch.zeros(1, self.in_channels, 1, 1))
        self.weight.data = F.softmax(self.weight.data.view(1, self.in_channels, -1), dim=-1).view(
            1, self.in_channels, self.kernel_size, self.kernel_size)
        self._tables = Kept(self._TABLE_SLOTS)
        self.fuse_gelu = False  # True: apply a GELU that follows inside the kernel

    def __setstate__(self, state):
        super().__setstate__(state)
        self._tables = Kept(self._TABLE_SLOTS)      # (also for modules pickled by earlier versions)

    # -- transfer-table cache: rebuilt when a parameter is modified in place or replaced
    def _table_for(self, h, w, device, which=0):
        """(table, weight as fp32) for padded planes h x w: 0 for every batch size; 1 the pair table and 2 the real-plane
        table alone, built when the first call that reads them comes (where both exist each is 0.5 to 1 times 8 C h w
        bytes, and a call reads one)."""
        weight, bias = self.weight, self.bias
        key = (h, w, self.scale, self.eps, which, _cabi.host().state(weight, bias))
        last = self._tables.last
        if last is not None and last[0] == key:
            return last[1]
        return self._tables.get(key, (weight, bias), lambda: _cabi.host().build_transfer(
            weight, bias, self.scale, self.eps, h, w, False, which))

    @property
    def biaseps(self):
        """lambda = sigmoid(bias - 9) + eps (`models/util_converse.py:147`)."""
        return torch.sigmoid(self.bias.detach() - 9.0) + self.eps

    def clear_cache(self):
        self._tables.clear()

    def _check_backend(self):
        host = _cabi.loaded_host()
        chosen = os.environ.get("CONVERSE2D_BACKEND") if host is None else host.backend()
        backend = (chosen or self.backend).lower()
        if backend == "pytorch":
            raise RuntimeError("Converse2D backend='pytorch' is not available: this build only has the "
                               "native sm_100a path")
        if backend not in ("auto", "cuda"):
            raise ValueError(f"backend must be 'auto' | 'cuda' | 'pytorch', got: {backend}")

    def forward(self, x, fuse_gelu=None):
        """`fuse_gelu`: apply the GELU that follows inside the kernel, for this call (None: the attribute decides)."""
        if fuse_gelu is None:
            fuse_gelu = self.fuse_gelu
        self._check_backend()
        if not x.is_cuda:
            raise RuntimeError("Converse2D backend='cuda' but the input is not a CUDA tensor.")
        shape = x.shape
        if len(shape) != 4 or shape[1] != self.in_channels:
            raise RuntimeError("x must be (B,%d,H,W)" % self.in_channels)
        p, host = self.padding, _cabi.host()
        h, w = shape[2] + 2 * p, shape[3] + 2 * p
        pairs = host.takes_pairs(shape[0], h, w, self.scale, shape[1])
        if torch.is_grad_enabled() and (x.requires_grad or self.weight.requires_grad or self.bias.requires_grad):
            # differentiable route (the reference is differentiable through torch.fft, converse2d.cpp:223)
            # its gradients read the real-plane table; so does the forward, but for the multi-pass pair kernels
            table, wf = self._table_for(h, w, x.device, 0 if pairs == 2 else 2)
            out = Converse2DFunction.apply(x, self.weight, self.bias, table, wf, self.kernel_size, self.scale,
                                           self.padding, self.padding_mode, self.eps)
            return F.gelu(out) if fuse_gelu else out
        which = 1 if pairs else 2
        table, wf = self._table_for(h, w, x.device, which)
        return host.converse2d(x, table, wf, self.kernel_size, self.scale, p, self.padding_mode, fuse_gelu, None, which)


def _with_gelu(conv, x):
    """conv(x) followed by the block's GELU, in one kernel.  Told by the call and not by the module's attribute, which
    another thread (or a hook that runs the block again) would see and reset; modules put in Converse2D's place that
    know only the attribute still get it."""
    if type(conv).forward is Converse2D.forward:
        return conv(x, fuse_gelu=True)
    conv.fuse_gelu = True
    try:
        return conv(x)
    finally:
        conv.fuse_gelu = False


class ConverseBlock(nn.Module):
    """`x + conv1(x)` then `x + conv2(x)` (`models/util_converse.py:253-293`); children and
    state-dict keys as in the reference (conv1.{0,1,3,5}, conv2.{0,1,3})."""

    def __init__(self, in_channels, out_channels, kernel_size=3, scale=1, padding=2, padding_mode="replicate",
                 eps=1e-5):
        super().__init__()
        self.conv1 = nn.Sequential(LayerNorm(in_channels, eps=1e-5, data_format="channels_first"),
                                   nn.Conv2d(in_channels, 2 * out_channels, 1, 1, 0),
                                   nn.GELU(),
                                   Converse2D(2 * out_channels, 2 * out_channels, kernel_size, scale=scale,
                                              padding=padding, padding_mode=padding_mode, eps=eps),
                                   nn.GELU(),
                                   nn.Conv2d(2 * out_channels, out_channels, 1, 1, 0))
        self.conv2 = nn.Sequential(LayerNorm(in_channels, eps=1e-5, data_format="channels_first"),
                                   nn.Conv2d(out_channels, 2 * out_channels, 1, 1, 0),
                                   nn.GELU(),
                                   nn.Conv2d(2 * out_channels, out_channels, 1, 1, 0))
        self._pack = Kept()          # 1x1 weights laid out for the kernels
        # True: bf16 tensors stay on the pair kernels and the layer-wise 1x1 kernels, so that a network that rounds every
        # activation to bf16 gives the outputs it always gave: its rounding amplifies the last bit of any value (random
        # weights: one pixel scaled by 1.0001 moves ConverseDnCNN's output by 1.3 %), and the block kernels' order of sums
        # moves it by 2.5 to 3.3 % (trained weights: 0.4 %).  They are no less accurate (2 x 96 x 128 against fp64: 3.08e-2
        # and 3.37e-2 in the fixed order with random weights, 2.3e-3 and 3.2e-3 with trained ones) and faster.  Set by
        # ConverseDnCNN.activation_dtype; a program that does not need the old outputs may reset it.
        self.fixed_order = False
        self._pair_table = Kept()

    def __setstate__(self, state):
        super().__setstate__(state)
        self._pack, self._pair_table = Kept(), Kept()
        self.__dict__.setdefault("fixed_order", False)

    def _branch1(self, x):
        c = self.conv1
        t = c[2](c[1](c[0](x)))
        return c[5](_with_gelu(c[3], t))     # c[4] runs inside the Converse2D kernel

    def _packed(self, params):
        """The 1x1 weights in the kernels' operand layout, laid out once per version of the parameters."""
        host = _cabi.host()
        key = (host.state(*params),)
        last = self._pack.last
        if last is not None and last[0] == key:
            return last[1]
        return self._pack.get(key, params, lambda: host.block_pack(*params))

    def _forward_trainable(self, x, alpha1=None, alpha2=None):
        """The block under autograd through the native kernels; None where they do not apply (other widths, dtypes or
        scales, hooked children, autocast, planes without a gradient kernel)."""
        c1, c2 = self.conv1._modules, self.conv2._modules
        conv = c1["3"]
        if not (BLOCK_FUSION and torch.is_grad_enabled() and x.is_cuda and x.dim() == 4 and x.size(1) == 64 and
                x.dtype == torch.float32 and c1["1"].out_channels == 128 and c1["5"].out_channels == 64 and
                conv.scale == 1 and not torch.is_autocast_enabled()):
            return None
        params = CF.block_parameters(c1["0"], c1["1"], c1["5"], alpha1, c2["0"], c2["1"], c2["3"], alpha2)
        given = [q for i, q in enumerate(params) if i not in (6, 13)] + [conv.weight, conv.bias]
        if any(q is None or q.dtype != torch.float32 or not q.is_cuda for q in given):
            return None
        for m in (self.conv1, self.conv2, *c1.values(), *c2.values()):
            if m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks:
                return None
        conv._check_backend()
        pack = self._packed(params)
        p, eps1, eps2, host = conv.padding, c1["0"].eps, c2["0"].eps, _cabi.host()
        h, w = x.shape[2] + 2 * p, x.shape[3] + 2 * p
        table, wf = conv._table_for(h, w, x.device, 0 if host.takes_pairs(x.shape[0], h, w, 1, conv.in_channels) == 2 else 2)
        x = x.contiguous()
        kept = host.block_train(x, table, wf, pack, conv.kernel_size, p, conv.padding_mode, eps1, eps2)
        if kept is None:
            return None
        return ConverseBlockFunction.apply(kept, x, conv.weight, conv.bias, table,
                                           (eps1, eps2, conv.eps, p, conv.padding_mode), *params)

    def _fusable(self, x):
        if torch.is_grad_enabled() and (x.requires_grad or any(q.requires_grad for q in self.parameters())):
            return False  # the fused block kernels are forward-only
        c1, c2 = self.conv1._modules, self.conv2._modules
        return (x.is_cuda and x.dim() == 4 and x.size(1) == 64 and c1["1"].out_channels == 128 and
                c1["5"].out_channels == 64 and c1["3"].scale == 1 and x.dtype in (torch.float32, torch.bfloat16) and
                c1["1"].bias is not None and c1["5"].bias is not None and c2["1"].bias is not None and
                c2["3"].bias is not None and BLOCK_FUSION)

    def _forward_fused(self, x, alpha1=None, alpha2=None):
        # LN+1x1+GELU, Converse2D(+GELU), 1x1+residual+LN+1x1+GELU+1x1+residual: one host call
        c1, c2 = self.conv1._modules, self.conv2._modules
        conv = c1["3"]
        if conv._forward_hooks or conv._forward_pre_hooks:
            return self._forward_layers(x, conv, alpha1, alpha2)
        if self.fixed_order and x.dtype == torch.bfloat16:
            return self._forward_fixed_order(x, conv, alpha1, alpha2)
        pack = self._packed(CF.block_parameters(c1["0"], c1["1"], c1["5"], alpha1, c2["0"], c2["1"], c2["3"], alpha2))
        conv._check_backend()
        shape, p, host = x.shape, conv.padding, _cabi.host()
        h, w = shape[2] + 2 * p, shape[3] + 2 * p
        which = 1 if host.takes_pairs(shape[0], h, w, 1, conv.in_channels) else 2
        table, wf = conv._table_for(h, w, x.device, which)
        return host.block(x, table, wf, pack, conv.kernel_size, p, conv.padding_mode, c1["0"].eps, c2["0"].eps, which)

    def _forward_fixed_order(self, x, conv, alpha1, alpha2):
        # (see `fixed_order`)
        c1, c2 = self.conv1, self.conv2
        h, w = x.size(2) + 2 * conv.padding, x.size(3) + 2 * conv.padding
        key = (h, w, conv.eps, x.device.index, _cabi.host().state(conv.weight, conv.bias))
        table, wf = self._pair_table.get(key, (conv.weight, conv.bias), lambda: CF.build_pair_transfer(
            conv.weight, conv.bias, conv.eps, h, w))
        t = CF.ln_pw_gelu(x, c1[0], c1[1])
        t = CF.pair_forward(t, table, wf, conv.kernel_size, conv.padding, conv.padding_mode, fuse_gelu=True)
        return CF.pw_res_mlp(t, x, c1[5], c2[0], c2[1], c2[3], alpha1, alpha2)

    def _forward_layers(self, x, conv, alpha1, alpha2):
        # the same kernels with Converse2D called as a module (someone hooked it)
        c1, c2 = self.conv1, self.conv2
        t = CF.ln_pw_gelu(x, c1[0], c1[1])
        t = _with_gelu(conv, t)
        return CF.pw_res_mlp(t, x, c1[5], c2[0], c2[1], c2[3], alpha1, alpha2)

    def forward(self, x):
        if self._fusable(x):
            return self._forward_fused(x)
        out = self._forward_trainable(x)
        if out is not None:
            return out
        with _exact_fp32():
            x = self._branch1(x) + x
            x = self.conv2(x) + x
        return x


class ConverseBlockAlphaVariant(ConverseBlock):
    """ConverseBlock with learned per-channel branch scales (`models/util_converse.py:297-323`)."""

    def __init__(self, in_channels, out_channels, kernel_size=3, scale=1, padding=2, padding_mode="replicate",
                 eps=1e-5):
        super().__init__(in_channels, out_channels, kernel_size, scale, padding, padding_mode, eps)
        self.alpha1 = nn.Parameter(torch.zeros((1, out_channels, 1, 1)), requires_grad=True)
        self.alpha2 = nn.Parameter(torch.zeros((1, out_channels, 1, 1)), requires_grad=True)

    def forward(self, x):
        if self._fusable(x):
            return self._forward_fused(x, self.alpha1, self.alpha2)
        out = self._forward_trainable(x, self.alpha1, self.alpha2)
        if out is not None:
            return out
        with _exact_fp32():
            x = self.alpha1 * self._branch1(x) + x
            x = self.alpha2 * self.conv2(x) + x
        return x
