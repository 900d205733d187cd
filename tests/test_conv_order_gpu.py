"""The tiled 3x3x3 kernel against the gathering one: the same products summed in
the same order, so the same bits.

A grid with small extents is mostly padding to the tiled kernel and runs in the
gathering one; the same grid repeated along y and z fills tiles and holds the
same periodic field.  The kernels that ran are read from the profiler, so that
a call that quietly took the other one fails."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(x0, x1, w, b, slope, f32):
    """The result and the names of the convolution kernels that made it."""
    from torch.profiler import ProfilerActivity, profile
    from lbflow_b200 import conv
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        y = conv.conv3_f32(x0, w, b) if f32 else conv.conv3(x0, w, b, slope, x1=x1)
        torch.cuda.synchronize()
    conv.check()
    names = [e.name for e in prof.events()]
    return y, {k for k in ('conv3_kernel', 'igemm_kernel') if any(k in n for n in names)}


@pytest.mark.parametrize('c0, c1, cout', [
    (8, 0, 16), (8, 0, 32), (8, 0, 64), (8, 0, 128), (8, 0, 200),     # two taps in a K step
    (16, 0, 16), (8, 8, 32), (16, 0, 64), (16, 0, 128),
    (32, 0, 32), (16, 16, 16), (32, 0, 64), (24, 8, 128), (48, 0, 24),
    (32, 32, 32), (48, 16, 64), (32, 32, 256),
])
def test_same_bits_from_both_kernels(c0, c1, cout):
    gen = torch.Generator().manual_seed(c0 + 3 * c1 + 5 * cout)
    x = torch.randn(2, 3, 4, 11, c0 + c1, generator=gen).to(torch.bfloat16).cuda()
    w = torch.randn(cout, c0 + c1, 3, 3, 3, generator=gen).cuda()
    b = torch.randn(cout, generator=gen).cuda()
    for slope, f32 in ((0.1, False), (None, False), (None, True)):
        if f32 and c1:
            continue
        out = []
        for y in (x, x.repeat(1, 2, 4, 1, 1)):
            s0 = y[..., :c0].contiguous()
            s1 = y[..., c0:].contiguous() if c1 else None
            out.append(_run(s0, s1, w, b, slope, f32))
        assert out[0][1] == {'igemm_kernel'} and out[1][1] == {'conv3_kernel'}
        assert torch.equal(out[0][0].repeat(1, 2, 4, 1, 1), out[1][0])


@pytest.mark.parametrize('channels', [24, 40, 56, 64])
def test_calls_that_stay_with_the_gathering_kernel(channels):
    """Channel counts whose K steps straddle taps unevenly, and 64 from one
    source, whose rows that kernel fetches whole, faster at every size."""
    x = torch.randn(1, 4, 16, 16, channels, device='cuda').to(torch.bfloat16)
    w = torch.randn(16, channels, 3, 3, 3, device='cuda')
    assert _run(x, None, w, None, None, False)[1] == {'igemm_kernel'}


def test_an_infinite_input_reaches_its_neighbours_only():
    """With one channel group the last tap shares its K step with zeros."""
    x = torch.zeros(1, 8, 16, 16, 8, device='cuda', dtype=torch.bfloat16)
    x[0, 4, 8, 8, 3] = float('inf')
    w = torch.ones(16, 8, 3, 3, 3, device='cuda')
    y, names = _run(x, None, w, None, None, True)
    assert names == {'conv3_kernel'}
    want = torch.zeros_like(y)
    want[0, 3:6, 7:10, 7:10] = float('inf')
    assert torch.equal(y, want)
