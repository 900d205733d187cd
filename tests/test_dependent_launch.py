"""Reads of the kernels that are launched with programmatic dependent launch.

Such a kernel starts while the previous kernels of its stream still run, so
whatever these write changes within its lifetime.  The read-only path (__ldg,
and loads through `const T* __restrict__`) is for data that does not change
while the kernel runs, and a compiler may move such a load above the wait for
the previous kernels.  The sources are therefore read with it in two cases
only: data that is fixed while an engine or batch steps, and kernels that are
launched without the attribute."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / 'lbflow_b200' / 'csrc'
SOURCES = ['kernels.cuh', 'color.cuh', 'color_step.cuh', 'resident.cuh', 'batch.cu', 'darcy.cu']

# Written at creation (or, the tile lists, by copies between launches).
FIXED = {'g.occ', 'g.coord', 'occ', 'coord', 'F.label', 'label', 'label_force', 'k.row', 'k.mask', 'k.base', 'row', 'mask',
         'base', 'z.bits', 'z.node', 'z.code', 'z.value', 'bits', 'node', 'code', 'value', 'film.bits', 'W.angle_id',
         'angle_id', 'angles', 'tib', 'geoms', 'tiles', 'tile_first', 'tile_count', 'mob'}
# Parameters of kernels launched without the attribute: initialisation, warm
# start, density increment, and the second pass of the batched sums.
ORDINARY = {'phase', 'fields', 'drho', 'partial'}


def _code(name):
    text = re.sub(r'/\*.*?\*/', ' ', (CSRC / name).read_text(), flags=re.S)
    return re.sub(r'//[^\n]*', '', text)


@pytest.mark.parametrize('name', SOURCES)
def test_read_only_loads_are_of_fixed_data(name):
    for m in re.finditer(r'__ldg\(\s*&?([\w.]+)', _code(name)):
        assert m.group(1) in FIXED, f'{name}: __ldg of {m.group(1)}'


@pytest.mark.parametrize('name', SOURCES)
def test_read_only_pointers_are_to_fixed_data(name):
    for m in re.finditer(r'\bconst\s+[\w:]+(?:\s+[\w:]+)?\s*\*\s*__restrict__\s+(\w+)', _code(name)):
        assert m.group(1) in FIXED | ORDINARY, f'{name}: const __restrict__ {m.group(1)}'


def test_the_ordinary_kernels_are_launched_without_the_attribute():
    launches = ''.join(_code(n) for n in SOURCES + ['scsp_launch.cu', 'color_launch.cu', 'engine.cu'])
    dependent = re.findall(r'launch_pdl(?:_shared)?\(\s*(\w+)', launches)
    assert dependent
    for kernel in ('scsp_init', 'scsp_init_eq', 'scsp_add_density', 'color_init', 'tile_sums', 'geom_sums', 'scsp_resident'):
        assert kernel not in dependent
