"""16-bit single-geometry steps, which take their pull sources from a table,
against the batched kernel, which looks them up: the same update on the same
values, so the fields are bitwise equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LABELS = {75: ('GV', 1e-5, 1, 0), 255: ('SD', 90.0, 0, 0)}


@pytest.mark.parametrize('shape, porosity', [
    ((3, 5, 1), 1.0), ((4, 3, 2), 0.8), ((1, 1, 33), 1.0),      # x and z wrap onto the voxel itself
    ((5, 4, 31), 0.7), ((5, 4, 32), 0.7), ((6, 7, 33), 0.7),    # around an occupancy word
    ((9, 40, 50), 0.5), ((130, 21, 20), 0.4),                   # tiles across plane ends
    ((2, 300, 300), 1.0), ((3, 270, 290), 0.9),                 # planes of more than 65,536 nodes
])
def test_table_matches_lookups(shape, porosity):
    from lbflow_b200 import Engine
    from lbflow_b200.batch import Batch
    g = np.where(np.random.default_rng(sum(shape)).random(shape) < porosity, 75, 255).astype(np.uint8)
    steps = 7
    with Engine(g, LABELS, tau=(0.9,), storage='fp16') as e:
        e.initialize()
        for _ in range(steps):
            e.step(1, macros=True)
        e.check()
        rho, _, u = e.macros()
    with Batch([g], [0.9], LABELS, storage='fp16') as b:
        b.initialize()
        b.step(steps, macros=True)
        b.check()
        r, v = b.macros(0)
    assert np.array_equal(rho, r) and np.array_equal(u, v)
