"""Backward passes of the operator's layers whose saved output or incoming
gradient is not the plain tensor the activation-gradient kernel reads: the same
gradients as from the plain one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(cin=16, cout=24, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(2, 4, 6, 8, cin, generator=g).to(torch.bfloat16).cuda().requires_grad_()
    w = (0.1 * torch.randn(cout, cin, 3, 3, 3, generator=g)).cuda().requires_grad_()
    b = torch.randn(cout, generator=g).cuda().requires_grad_()
    gy = torch.randn(2, 4, 6, 8, cout, generator=g).to(torch.bfloat16).cuda()
    return x, w, b, gy


def _shifted(t):
    """t at an address that is no multiple of 16 bytes."""
    s = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    return s.copy_(t)


FORMS = {
    'strided': lambda t: t.permute(0, 4, 1, 2, 3).contiguous().permute(0, 2, 3, 4, 1),
    'misaligned': _shifted,
    'float': lambda t: t.float(),
}


@pytest.mark.parametrize('form', FORMS)
def test_saved_output_from_hooks(form):
    from lbflow_b200 import conv
    x, w, b, gy = _inputs()
    want = torch.autograd.grad(conv.conv3(x, w, b, 0.1), (x, w, b), gy)

    def unpack(t):
        return FORMS[form](t) if t.shape == gy.shape else t

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        y = conv.conv3(x, w, b, 0.1)
        got = torch.autograd.grad(y, (x, w, b), gy)
    conv.check()
    for name, a, c in zip('xwb', want, got):
        if name == 'b':            # sums in another order in torch's form
            assert torch.allclose(a, c, rtol=1e-5, atol=1e-5 * float(gy.float().abs().sum(dim=(0, 1, 2, 3)).max()))
        else:
            assert torch.equal(a, c)


@pytest.mark.parametrize('form', ['strided', 'misaligned'])
def test_incoming_gradient(form):
    from lbflow_b200 import conv
    x, w, b, gy = _inputs(seed=1)
    y = conv.conv3(x, w, b, 0.1)
    want = torch.autograd.grad(y, (x, w, b), gy, retain_graph=True)
    got = torch.autograd.grad(y, (x, w, b), FORMS[form](gy))
    for a, c in zip(want, got):
        assert torch.equal(a, c)


@pytest.mark.parametrize('slope', [0.1, None])
def test_bias_gradient_is_differentiable_in_the_incoming_one(slope):
    from lbflow_b200 import conv
    x, w, b, gy = _inputs(seed=2)
    y = conv.conv3(x, w, b, slope)
    gy = gy.requires_grad_()
    gb, = torch.autograd.grad(y, b, gy, create_graph=True)
    d, = torch.autograd.grad(gb.sum(), gy)
    factor = torch.where(y > 0, 1.0, slope) if slope is not None else torch.ones_like(y)
    assert torch.equal(d, factor.to(torch.bfloat16))


def test_a_weight_with_the_negative_bit():
    """The imaginary part of a conjugate view is its negative, unresolved."""
    from lbflow_b200 import conv
    x, w, b, _ = _inputs(seed=3)
    z = torch.complex(torch.zeros_like(w.detach()), w.detach()).conj().imag
    assert z.is_neg()
    assert torch.equal(conv.conv3(x, z, b, None), conv.conv3(x, -w, b, None))
