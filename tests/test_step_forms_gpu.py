"""Steps launched one by one against the reference's outputs: calls of several
steps on geometries this small run in the resident launch, which leaves the
ordinary step kernel to this file and to bitwise comparisons with that form."""
import pytest

import test_parity_gpu as parity
from cases import golden_cases
from conftest import fluid_mask, load_golden

pytestmark = pytest.mark.gpu

CASES = [c for c in golden_cases() if c['model'] != 'color' and c['steps'] <= 2000]


@pytest.mark.parametrize('case', CASES, ids=[c['name'] for c in CASES])
def test_single_steps_match_reference(case):
    gold = load_golden(case['name'])
    fl = fluid_mask(case)
    fl3 = fl if fl.ndim == 3 else fl[None]
    with parity.engine_for(case) as e:
        e.initialize()
        before = e.device_bytes
        for _ in range(case['steps'] - 1):
            e.step(1)
        e.step(1, macros=True)
        e.check()
        assert e.device_bytes == before         # no resident launch
        f = e.populations()
        rtol = parity.population_tolerance(case, case['steps'])
        parity.assert_populations_close(f, gold['populations'].reshape(f.shape), fl3, rtol)
        parity.assert_macros_close(e.macros(), parity.golden_macros(case, gold), fl3, rtol)
