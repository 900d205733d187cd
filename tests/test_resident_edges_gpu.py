"""Which calls take the resident launch of several steps, and what it does at its
edges: a wait that runs out, several engines at once, a captured stream."""
import ctypes
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LABELS = {75: ('GV', 1e-5, 1, 0), 10: ('PB', 1.0005, 1, 0), 11: ('PB', 0.9995, 2, 0), 255: ('SD', 90.0, 0, 0)}


def _medium(shape, porosity=0.6, seed=3):
    return np.where(np.random.default_rng(seed).random(shape) < porosity, 75, 255).astype(np.uint8)


def _engine(g, storage='fp64', collision='MRT'):
    from lbflow_b200 import Engine
    return Engine(g, LABELS, collision=collision, tau=(0.9,), storage=storage)


def _fields(e):
    e.check()
    rho, _, u = e.macros()
    return rho, u, e.populations()


def _word_bytes(e, storage):
    q = 19 if e.dims == 3 else 9
    return 2 * (q - 1) * ((e.fluid_nodes + 63) // 64 * 64) * (16 if storage == 'fp64' else 8)


# The words of a resident launch show in the engine's device memory.
@pytest.mark.parametrize('storage, shape, steps, resident', [
    ('fp64', (1, 3, 11), 2, True), ('fp64', (13, 20, 37), 38, True), ('fp64', (13, 20, 37), 1, False),
    ('fp32', (13, 20, 37), 3, True), ('fp16', (13, 20, 37), 3, True), ('bf16', (13, 20, 37), 3, True),
    ('bfp16', (13, 20, 37), 3, False),
    ('fp64', (40, 48), 9, True), ('fp32', (40, 48), 9, True), ('fp16', (40, 48), 9, True),
])
def test_which_calls_are_resident(storage, shape, steps, resident):
    with _engine(_medium(shape, 0.9), storage) as e:
        e.initialize()
        before = e.device_bytes
        e.step(steps)
        assert e.device_bytes - before == (_word_bytes(e, storage) if resident else 0)
        e.check()


@pytest.mark.parametrize('storage, most', [('fp64', 16), ('fp32', 28), ('fp16', 28), ('bf16', 28)])
def test_the_largest_resident_geometry(storage, most):
    """`most` warps per SM: one more node than the GPU holds is stepped launch by
    launch."""
    import torch
    nodes = torch.cuda.get_device_properties(0).multi_processor_count * most * 32
    g = np.full((nodes // 2048 + 2, 32, 64), 255, np.uint8)
    for extra in (0, 1):
        g.ravel()[:nodes + extra] = 75
        with _engine(g, storage) as e:
            e.initialize()
            before = e.device_bytes
            e.step(3)
            e.check()
            assert (e.device_bytes > before) == (extra == 0)


def test_boundaries_and_kept_solids_step_launch_by_launch():
    g = _medium((9, 10, 24), 0.9)
    for keep in (False, True):
        b = g.copy()
        if not keep:
            b[..., 0], b[..., -1] = 10, 11
        with _engine(b, collision='SRT') as e:
            if keep:
                e.keep_solid_populations()
            e.initialize()
            before = e.device_bytes
            e.step(4)
            e.check()
            assert e.device_bytes == before


@pytest.mark.parametrize('storage, shape', [('fp64', (48, 48, 48)), ('fp32', (48, 48, 48)), ('fp64', (300, 300))])
def test_a_wait_that_runs_out(storage, shape):
    """With no patience at all the launch returns early, says so, and lets later
    calls return too; a new state on the same engine is a healthy one again."""
    from lbflow_b200 import LbfError
    g = _medium(shape)
    with _engine(g, storage) as healthy:
        healthy.initialize()
        healthy.step(60, macros=True)
        want = _fields(healthy)
    with _engine(g, storage) as e:
        e.initialize()
        e.step(20)
        e.check()
        assert e._lib.lbf_set_wait_limit(e._h, ctypes.c_uint64(0)) == 0
        t = time.perf_counter()
        e.step(400)
        with pytest.raises(LbfError, match='gave up waiting'):
            e.check()
        e.step(3000)
        with pytest.raises(LbfError, match='gave up waiting'):
            e.check()
        assert time.perf_counter() - t < 1.0
        assert e._lib.lbf_set_wait_limit(e._h, ctypes.c_uint64(4000000000)) == 0
        e.initialize()
        e.step(60, macros=True)
        for a, b in zip(want, _fields(e)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize('shape', [(24, 30, 36), (32, 37, 64)])
def test_engines_in_several_threads(shape):
    """Each launch of the second size fills the GPU on its own."""
    media = [np.full(shape, 75, np.uint8) if k == 0 else _medium(shape, 0.97, k) for k in range(3)]

    def run(g, out, k):
        with _engine(g) as e:
            e.initialize()
            for n in (50, 3, 300, 1, 1100, 2):
                e.step(n, macros=True)
            out[k] = _fields(e)

    alone, together = {}, {}
    for k, g in enumerate(media):
        run(g, alone, k)
    threads = [threading.Thread(target=run, args=(g, together, k)) for k, g in enumerate(media)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(3):
        for a, b in zip(alone[k], together[k]):
            assert np.array_equal(a, b)


@pytest.mark.parametrize('storage', ['fp64', 'fp32'])
def test_a_captured_call_replays(storage):
    """While its stream is captured an engine steps launch by launch; a replay
    repeats the steps from where the populations stand."""
    g = _medium((13, 20, 37))
    with _engine(g, storage) as e:
        e.initialize()
        e.step(16, macros=True)
        want = _fields(e)
    rt = ctypes.CDLL('libcudart.so.12')
    with _engine(g, storage) as e:
        e.initialize()
        e.step(2)                                       # resident, before the capture
        e.synchronize()
        stream = ctypes.c_void_p(e.stream)
        graph, exe = ctypes.c_void_p(), ctypes.c_void_p()
        assert rt.cudaStreamBeginCapture(stream, 1) == 0
        e.step(4, macros=True)                          # an even number: the buffers end where they began
        assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) == 0
        assert rt.cudaGraphInstantiateWithFlags(ctypes.byref(exe), graph, ctypes.c_ulonglong(0)) == 0
        for _ in range(3):
            assert rt.cudaGraphLaunch(exe, stream) == 0
        e.synchronize()
        e.step(2, macros=True)                          # resident again, after it
        got = _fields(e)
        assert rt.cudaGraphExecDestroy(exe) == 0 and rt.cudaGraphDestroy(graph) == 0
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
