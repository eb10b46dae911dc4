"""What a module keeps between calls (transfer tables, packed 1x1 weights) follows its parameters."""
import pytest
import torch


def _rel(a, r):
    return float((a.double() - r.double()).norm() / r.double().norm())


def test_inference_tensors_have_no_state():
    from conversenet_b200 import _cabi
    with torch.inference_mode():
        t = torch.zeros(3)
    assert _cabi.host().state(torch.zeros(3), None, t) is None
    assert _cabi.host().state(torch.zeros(3), None) is not None


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_modules_made_in_inference_mode_follow_their_parameters(dtype):
    from conversenet_b200 import Converse2D, ConverseBlock

    def change(m):
        for i, q in enumerate(m.parameters()):
            q.add_(0.05 * (i + 1))

    for make, C in ((lambda: Converse2D(8, 8, 3, padding=1), 8), (lambda: ConverseBlock(64, 64, 3, 1, 1), 64)):
        for fixed in (False, True):
            torch.manual_seed(5)
            ordinary = make().cuda().eval()
            x = torch.randn(2, C, 20, 17, device="cuda").to(dtype)
            with torch.inference_mode():
                m = make().cuda().eval()
                m.load_state_dict(ordinary.state_dict())
                m.fixed_order = ordinary.fixed_order = fixed
                first = m(x)
                change(m)
                second = m(x)
            with torch.no_grad():
                assert torch.equal(first, ordinary(x))
                change(ordinary)
                assert torch.equal(second, ordinary(x))
            assert _rel(second, first) > 1e-3
