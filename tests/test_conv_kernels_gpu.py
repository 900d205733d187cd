"""The tiled 3x3x3 kernel, the weight packing and the activation-gradient pass
of the warm-start operator against torch in FP64 (convolution) or the same
operations in torch (the other two)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize('dims, c0, c1, cout', [
    ((1, 4, 16, 8), 16, 0, 16),      # one tile of 8 x 16 x 4 voxels
    ((2, 8, 30, 15), 8, 0, 16),      # half an operand of channels, ragged x and y
    ((1, 7, 31, 23), 24, 8, 8),      # two sources, ragged in all axes, 8 outputs
    ((1, 9, 16, 40), 40, 0, 24),     # channels between the compiled widths
    ((1, 4, 32, 17), 32, 32, 64),    # widest input
    ((2, 4, 15, 16), 64, 0, 128),    # widest output
    ((1, 5, 16, 24), 16, 0, 136),    # more than one block of outputs
])
@pytest.mark.parametrize('slope', [0.1, None])
def test_conv3_tiles(dims, c0, c1, cout, slope):
    """One bf16 rounding (2^-9) of the result on top of FP32 accumulation."""
    from lbflow_b200 import conv
    cin = c0 + c1
    x = _rand(*dims, cin, seed=1)
    w = _rand(cout, cin, 3, 3, 3, scale=(27 * cin) ** -0.5, seed=2).float()
    b = 0.1 * torch.randn(cout, generator=torch.Generator().manual_seed(3))
    ref = F.conv3d(F.pad(x.double().permute(0, 4, 1, 2, 3), (1, 1, 1, 1, 1, 1), mode='circular'), w.double(), b.double())
    lin = ref.permute(0, 2, 3, 4, 1)
    ref = torch.where(lin > 0, lin, slope * lin) if slope is not None else lin
    xs = x.cuda()
    y = conv.conv3(xs[..., :c0].contiguous(), w.cuda(), b.cuda(), slope, x1=xs[..., c0:].contiguous() if c1 else None)
    conv.check()
    err = (y.double().cpu() - ref).abs()
    assert torch.all(err <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max())
    if slope is None and not c1:
        y = conv.conv3_f32(xs, w.cuda(), b.cuda())
        assert (y.double().cpu() - ref).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize('shape, order, split, flip', [
    ((16, 8, 3, 3, 3), (0, 2, 3, 4, 1), 1, False), ((24, 40, 3, 3, 3), (1, 2, 3, 4, 0), 1, True),
    ((32, 16, 2, 2, 2), (2, 3, 4, 1, 0), 4, False), ((136, 8, 3, 3, 3), (0, 2, 3, 4, 1), 1, False),
])
def test_pack_weight(shape, order, split, flip):
    from lbflow_b200 import conv
    w = torch.randn(*shape, device='cuda')
    v = (w.flip(2, 3, 4) if flip else w).permute(order)
    n = 1
    for d in v.shape[:split]:
        n *= d
    p = conv._pack(w, order, split, flip)
    assert (p.n, p.k) == (n, w.numel() // n)
    assert torch.equal(p.data, conv.pack_weight(v.reshape(n, -1)))


@pytest.mark.parametrize('rows, c', [(1, 8), (7, 24), (1000, 64), (65537, 16), (33, 2048)])
@pytest.mark.parametrize('slope', [0.1, None])
def test_act_grad(rows, c, slope):
    """The masked gradient exactly; the channel sums to FP32 accumulation
    (2^-23 per addition of at most rows terms, pessimistically 1e-5 of the sum of magnitudes)."""
    from lbflow_b200 import conv
    gy = _rand(1, rows, 1, 1, c, seed=1).cuda()
    y = _rand(1, rows, 1, 1, c, seed=2).cuda()
    y[0, 0, 0, 0, 0] = 0.0
    want = (gy.float() * torch.where(y > 0, 1.0, slope)).to(torch.bfloat16) if slope is not None else gy
    out, gb = conv._act_grad(gy, y, slope, True)
    assert torch.equal(out, want)
    ref = want.double().sum(dim=(0, 1, 2, 3))
    assert torch.all((gb.double() - ref).abs() <= 1e-5 * want.double().abs().sum(dim=(0, 1, 2, 3)))
    # A view that is neither contiguous nor 16-byte aligned.
    wide = torch.cat([gy, gy], dim=-1)[..., 4:4 + c]
    wide2 = wide.contiguous()
    assert torch.equal(conv._act_grad(wide, y, slope, False)[0], conv._act_grad(wide2, y, slope, False)[0])
