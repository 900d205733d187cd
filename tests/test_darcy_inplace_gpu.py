"""The block pressure solve with its result written over the mobilities."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape', [(8, 8, 8), (16, 12, 20), (32, 32, 32)])
def test_in_place(shape):
    from lbflow_b200 import warmstart as W
    mob = torch.exp(torch.randn(shape, generator=torch.Generator().manual_seed(5), dtype=torch.float64)).cuda()
    want, it = W.darcy_pressure_device(mob, 1e-5, 2, rtol=1e-8, max_iter=200)
    from lbflow_b200 import library
    lib = library()
    both, got_it = mob.clone(), ctypes.c_uint32()
    rc = lib.lbf_darcy_pressure(ctypes.c_void_p(both.data_ptr()), *shape, 2.0, 1e-5, 1e-8, 200,
                                ctypes.c_void_p(both.data_ptr()), ctypes.byref(got_it),
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and got_it.value == it and it > 0
    assert torch.equal(both, want)
