"""New values of a matrix given as device memory through the C ABI, without the
fence the Python layer puts around the call."""
import numpy as np
import pytest
import torch

from spmv_b200 import _lib, gen
from spmv_b200._lib import ptr_array
from helpers import build

pytestmark = pytest.mark.gpu


def set_device_values(M, tensors):
    _lib.call("spmv_matrix_set_values", M.handle, _lib.MEMORY_DEVICE,
              ptr_array([t.data_ptr() for t in tensors]))


def test_values_still_being_computed_on_the_default_stream(cuda_device):
    W = gen.workload("c1", 60)
    comm, cm, rm, M, D = build(W, 3)
    new = [np.random.default_rng(q).standard_normal(len(D.blocks[q][2])) for q in range(3)]
    src = [torch.from_numpy(v).cuda() for v in new]
    vals = [torch.zeros_like(v) for v in src]
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)  # about 10 ms
    for v, s in zip(vals, src):
        v.copy_(s)
    set_device_values(M, vals)
    for q in range(3):
        np.testing.assert_array_equal(M.mat(q)[2], new[q])


def test_the_callers_pointer_shows_new_device_values(cuda_device):
    import ctypes as C
    W = gen.workload("c1", 40)
    comm, cm, rm, M, D = build(W, 2)
    rp, ci, va = C.POINTER(C.c_int32)(), C.POINTER(C.c_int32)(), C.c_void_p()
    _lib.call("spmv_matrix_csr", M.handle, 1, C.byref(rp), C.byref(ci), C.byref(va))
    held = np.ctypeslib.as_array(C.cast(va, C.POINTER(C.c_double)), (len(D.blocks[1][2]),))
    np.testing.assert_array_equal(held, D.blocks[1][2])
    for seed in (1, 2):
        new = [np.random.default_rng(seed + q).standard_normal(len(D.blocks[q][2]))
               for q in range(2)]
        M.set_values([torch.from_numpy(v).cuda() for v in new])
        np.testing.assert_array_equal(held, new[1])
