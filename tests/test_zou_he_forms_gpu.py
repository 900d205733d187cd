"""Boundary nodes updated inside the step's launch and in a launch of their own:
the same update, so the same bits.

A small medium between pressure planes takes the first form; repeated along the
periodic y and z it has the same fields and enough nodes for the second.  Which
kernels ran is read from the profiler."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LABELS = {75: ('GV', 2e-6, 1, 0), 76: ('GV', 1e-6, 3, 0), 10: ('PB', 1.0005, 1, 0), 11: ('PB', 0.9995, 2, 0),
          12: ('VB', 1e-4, 1, 0), 255: ('SD', 90.0, 0, 0)}


def _medium(shape, inlet):
    rng = np.random.default_rng(sum(shape))
    g = np.where(rng.random(shape) < 0.8, np.where(rng.random(shape) < 0.5, 75, 76), 255).astype(np.uint8)
    g[..., :2] = 75
    g[..., -2:] = 75
    g[..., 0], g[..., -1] = inlet, 11
    return g


def _fields(g, storage, collision):
    """Fields after some steps, and whether the boundary pass was launched."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    from lbflow_b200 import Engine
    with Engine(g, LABELS, collision=collision, tau=(0.9,), storage=storage) as e:
        e.initialize()
        e.step(6)
        e.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            e.step(4, adjacent=True)
            e.step(1, macros=True)
            e.synchronize()
            torch.cuda.synchronize()
        e.check()
        rho, _, u = e.macros()
        conv = e.convergence()
    return rho, u, conv, any('scsp_zou_he_pass' in k.name for k in prof.events())


@pytest.mark.parametrize('inlet', [10, 12])
@pytest.mark.parametrize('storage, shape, times', [
    ('fp64', (12, 16, 33), (14, 12)), ('fp32', (12, 16, 33), (18, 16)), ('fp64', (41, 600), (48,)), ('fp16', (12, 16, 33), (14, 12)),
])
@pytest.mark.parametrize('collision', ['SRT', 'MRT'])
def test_both_forms_agree(storage, shape, times, inlet, collision):
    g = _medium(shape, inlet)
    large = np.tile(g, times + (1,))
    rho, u, conv, apart = _fields(g, storage, collision)
    rho_l, u_l, conv_l, apart_l = _fields(large, storage, collision)
    assert not apart and apart_l == (storage != 'fp16')
    if storage == 'fp16':
        return                      # rounding streams follow the node numbers
    assert np.array_equal(np.tile(rho, times + (1,)), rho_l)
    assert np.array_equal(np.tile(u, (1,) + times + (1,)), u_l)
    # Sums of the velocity's change: the same nodes in another order.
    assert np.allclose(np.asarray(conv)[:3] * np.prod(times), np.asarray(conv_l)[:3], rtol=1e-9)
