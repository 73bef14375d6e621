"""What the entry points allocate on the device."""
import ctypes

import numpy as np
import pytest

from oracle import quasi_oracle as qo

pytestmark = pytest.mark.gpu


def test_instance_size():
    """Fields of a 256x256x256 instance: 24 float and 12 double ones in the FP32
    form, 36 double ones in FP64; 16 MiB for tables, graphs and the rest."""
    import torch

    import smaiso_quasi_b200 as q
    cells = 256 ** 3
    q.Simulation(q.default_config("quasi", 16, 16, 32))   # the library and its kernels are loaded
    for precision, per_cell in (("fp32", 24 * 4 + 12 * 8), ("fp64", 36 * 8)):
        warm = q.Simulation(q.default_config("quasi", 256, 256, 256, precision=precision))
        del warm
        free = torch.cuda.mem_get_info()[0]
        s = q.Simulation(q.default_config("quasi", 256, 256, 256, precision=precision))
        used = free - torch.cuda.mem_get_info()[0]
        del s
        assert used <= per_cell * cells + (16 << 20), (precision, used / cells)


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
