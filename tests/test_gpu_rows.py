"""Row transforms (the z pass) at the lengths and row counts where the lane
placement changes: every z length, with the fewest rows a grid may have and with
a row count that leaves the last CTA partly empty, against the oracle's
transforms.  Tolerances are those of the other transform tests: a few ulp times
log2(N)."""
import numpy as np
import pytest

from oracle import quasi_oracle as qo

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-14, "fp32": 2e-6}


@pytest.mark.parametrize("nz", [16, 32, 64, 96, 128, 192, 256, 512])
@pytest.mark.parametrize("rows", [(8, 8), (96, 32)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_row_lengths(nz, rows, precision):
    import smaiso_quasi_b200 as q
    grid = (*rows, nz)
    a = np.random.default_rng(nz).standard_normal(grid)
    for plan in ("CT", "iCT", "STz", "iSTz"):
        ref = qo.r2r3d(a, qo.PLAN_KINDS[plan])
        got = q.R2RPlan(*grid, plan, precision=precision).execute_host(a)
        err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
        assert err < TOL[precision], (plan, err)
