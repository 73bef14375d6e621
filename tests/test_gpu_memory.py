"""What the entry points allocate on the device."""
import ctypes

import numpy as np
import pytest

from oracle import quasi_oracle as qo

pytestmark = pytest.mark.gpu


def pool_high(reset=False):
    """Most bytes ever taken from the device's default memory pool."""
    cu = ctypes.CDLL("libcuda.so.1")
    pool, v = ctypes.c_void_p(), ctypes.c_uint64(0)
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    used_high = 8   # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    if reset:
        assert cu.cuMemPoolSetAttribute(pool, used_high, ctypes.byref(v)) == 0
    assert cu.cuMemPoolGetAttribute(pool, used_high, ctypes.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("grid", [(16, 32, 64), (16, 16, 512), (16, 512, 16), (512, 16, 32), (512, 8, 512)])
@pytest.mark.parametrize("plan", ["CT", "iCT", "STx", "STy", "STz", "iSTx", "iSTy", "iSTz"])
def test_float_pairs_are_transformed_in_place(grid, plan):
    """Floats that are 8- but not 16-byte aligned take no buffer, whatever the
    lengths.  2e-6: the tolerance of the float transforms."""
    import torch

    import smaiso_quasi_b200 as q
    a = np.random.default_rng(7).standard_normal(grid)
    ref = qo.r2r3d(a, qo.PLAN_KINDS[plan])
    p = q.R2RPlan(*grid, plan, precision="fp32")
    x = torch.empty(a.size + 2, dtype=torch.float32, device="cuda")[2:]
    x.copy_(torch.from_numpy(a.astype(np.float32)).reshape(-1))
    torch.cuda.synchronize()
    pool_high(reset=True)
    p.execute_device(x.data_ptr())
    assert pool_high() == 0
    got = x.double().cpu().numpy().reshape(grid)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 2e-6
