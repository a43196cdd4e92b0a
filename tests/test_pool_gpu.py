"""Large temporaries go back to the device: after a synchronisation the default memory pool holds at most
8 GiB beside what is in use."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
_RESERVED_MEM_CURRENT, _USED_MEM_CURRENT = 5, 7  # CUmemPool_attribute


def _idle_bytes():
    drv, pool = C.CDLL("libcuda.so.1"), C.c_void_p()
    assert drv.cuDeviceGetDefaultMemPool(C.byref(pool), C.c_int(torch.cuda.current_device())) == 0
    val = {}
    for attr in (_RESERVED_MEM_CURRENT, _USED_MEM_CURRENT):
        v = C.c_uint64(0)
        assert drv.cuMemPoolGetAttribute(pool, attr, C.byref(v)) == 0
        val[attr] = v.value
    return val[_RESERVED_MEM_CURRENT] - val[_USED_MEM_CURRENT]


def test_idle_blocks(mr, cuda):
    rng = np.random.default_rng(81)
    trj = (rng.random((3, 500, 2)) - 0.5).astype(np.float32)
    U = rng.standard_normal((2, 3)).astype(np.float32)
    for _ in range(2):
        mr.NFFTNormalOp((144, 144, 144), trj, U).close()  # 12 GB of grids
    torch.cuda.synchronize()
    assert _idle_bytes() <= 8 << 30
