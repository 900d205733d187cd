"""Steps of one resident launch (engine.step(n > 1) of a geometry that fits on
the GPU at once) against the same steps launched one by one.  Both evaluate the
same expressions on the same values, so populations and fields are bitwise
equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(geometry, storage, collision, chunks):
    from lbflow_b200 import Engine
    labels = {75: ('GV', 1e-5, 1, 0), 76: ('GV', 3e-5, 3, 0), 255: ('SD', 90.0, 0, 0)}
    with Engine(geometry, labels, collision=collision, tau=(0.9,), storage=storage) as e:
        e.initialize()
        for n in chunks:
            e.step(n, macros=True, adjacent=True)
        e.check()
        rho, _, u = e.macros()
        return e.populations(), rho, u, e.convergence()


def _geometry(shape, porosity, two_forces):
    rng = np.random.default_rng(sum(shape))
    g = np.where(rng.random(shape) < porosity, 75, 255).astype(np.uint8)
    if two_forces:
        g[(g == 75) & (rng.random(shape) < 0.5)] = 76
    return g


@pytest.mark.parametrize('storage', ['fp64', 'fp32', 'fp16', 'bf16'])
@pytest.mark.parametrize('shape, porosity, collision', [
    ((1, 1, 1), 1.0, 'MRT'),          # one node, its own neighbour in every direction
    ((1, 1, 31), 1.0, 'SRT'), ((1, 3, 11), 1.0, 'MRT'), ((4, 4, 2), 1.0, 'MRT'),   # around one warp
    ((13, 20, 37), 0.6, 'MRT'),       # ragged rows, isolated nodes
    ((40, 48), 0.5, 'SRT'), ((5, 33), 1.0, 'MRT'),                                 # D2Q9
])
def test_resident_steps_match_single_steps(storage, shape, porosity, collision):
    g = _geometry(shape, porosity, two_forces=True)
    if not (g != 255).any():
        pytest.skip('no pore voxel')
    one = _state(g, storage, collision, [1] * 38)
    many = _state(g, storage, collision, [2, 13, 3, 19, 1])
    for a, b in zip(one, many):
        assert np.array_equal(a, b)


@pytest.mark.parametrize('storage, shape', [
    ('fp64', (32, 37, 64)), ('fp64', (32, 37, 65)),        # 148 SMs x 16 warps, and more than fit
    ('fp32', (64, 37, 56)), ('fp16', (64, 37, 56)),        # 148 SMs x 28 warps
    ('fp64', (296, 320)), ('fp32', (296, 512)),            # D2Q9: 20 and 32 warps per SM
])
def test_largest_geometries(storage, shape):
    g = np.full(shape, 75, np.uint8)
    g[..., 0] = 76
    one = _state(g, storage, 'MRT', [1] * 9)
    many = _state(g, storage, 'MRT', [9])
    for a, b in zip(one, many):
        assert np.array_equal(a, b)


@pytest.mark.parametrize('storage', ['fp64', 'fp16'])
@pytest.mark.parametrize('steps', [1023, 1024, 1025, 2049])
def test_calls_of_several_launches(storage, steps):
    """A resident launch takes at most 1,024 steps and at least two."""
    g = _geometry((3, 5, 7), 0.9, two_forces=False)
    one = _state(g, storage, 'MRT', [1] * steps)
    many = _state(g, storage, 'MRT', [steps])
    for a, b in zip(one[:3], many[:3]):
        assert np.array_equal(a, b)
