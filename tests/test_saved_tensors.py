"""What the training forwards keep for their backwards: saved tensors, that hooks see and that the backward releases."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(scale):
    from conversenet_b200 import Converse2D
    return Converse2D(6, 6, 3, scale=scale, padding=2).cuda(), 6


def _block(_):
    from conversenet_b200 import ConverseBlock
    return ConverseBlock(64, 64, 3, 1, 2, "circular").cuda(), 64


CASES = [(_layer, 1), (_layer, 2), (_block, 1)]


def _run(m, x):
    y = m(x)
    return y, torch.autograd.grad(y, [x] + list(m.parameters()), torch.ones_like(y), retain_graph=True)


@pytest.mark.parametrize("make,scale", CASES)
def test_hooks_see_every_kept_plane_and_gradients_follow_them(make, scale):
    torch.manual_seed(scale)
    m, C = make(scale)
    x = torch.randn(2, C, 24, 20, device="cuda", requires_grad=True)
    ref = _run(m, x)[1]
    seen = []

    def pack(t):
        seen.append(t.numel() if t.is_floating_point() else 0)
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        got = _run(m, x)[1]
    # the input; r at scale 2 (24 + 4 rows of 20 + 4); t1, z1, u, x1, z3 of a block
    pixels = 2 * 24 * 20
    want = C * pixels + (0 if scale == 1 else 2 * C * 28 * 24)
    if make is _block:
        want = (64 + 4 * 128 + 64) * pixels
    assert sum(seen) >= want
    for a, r in zip(got, ref):
        assert torch.equal(a, r)


@pytest.mark.parametrize("make,scale", CASES[1:])        # a layer at scale 1 keeps nothing of its own
def test_backward_releases_what_the_forward_kept(make, scale):
    m, C = make(scale)
    x = torch.randn(2, C, 64, 64, device="cuda", requires_grad=True)
    loss = m(x).sum()
    loss.backward()                      # warm-up: gradients, tables, packed weights
    del loss
    base = torch.cuda.memory_allocated()
    loss = m(x).sum()
    kept = torch.cuda.memory_allocated() - base
    loss.backward()
    assert kept > x.numel() * 4          # something was kept
    assert torch.cuda.memory_allocated() - base <= 4096 and loss.grad_fn is not None


def test_a_plane_that_no_kernel_reads_is_not_kept():
    from conversenet_b200 import Converse2D
    m = Converse2D(4, 4, 3, scale=5, padding=1).cuda()         # parameter gradients through the torch.fft restatement
    x = torch.randn(1, 4, 62, 62, device="cuda")
    m(x)
    base = torch.cuda.memory_allocated()
    y = m(x)
    assert torch.cuda.memory_allocated() - base <= y.numel() * 4 + 4096


@pytest.mark.parametrize("make,scale", CASES)
def test_a_second_derivative_is_refused(make, scale):
    m, C = make(scale)
    x = torch.randn(1, C, 12, 10, device="cuda", requires_grad=True)
    y = m(x)
    gx, = torch.autograd.grad(y.square().sum(), x, create_graph=True)
    with pytest.raises(RuntimeError):
        (gx.square().sum() + 0.0 * x.sum()).backward()


def test_checkpointed_block_gives_the_same_gradients():
    from torch.utils.checkpoint import checkpoint
    m, C = _block(1)
    x = torch.randn(1, C, 16, 18, device="cuda", requires_grad=True)
    ref = _run(m, x)[1]
    y = checkpoint(m, x, use_reentrant=False)
    got = torch.autograd.grad(y, [x] + list(m.parameters()), torch.ones_like(y))
    for a, r in zip(got, ref):
        assert torch.equal(a, r)
