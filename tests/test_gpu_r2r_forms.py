"""Transforms above the size whose column passes run without tensor copies (16 MB):
every length that a column pass of such a field can have, sine and cosine kinds
both ways.  Tolerances are those of the smaller transforms."""
import numpy as np
import pytest

from oracle import quasi_oracle as qo

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-14, "fp32": 2e-6}


@pytest.mark.parametrize("grid,precision", [((16, 512, 512), "fp64"), ((512, 16, 512), "fp64"), ((32, 256, 512), "fp64"),
                                            ((256, 32, 512), "fp64"), ((64, 192, 192), "fp64"), ((192, 64, 256), "fp64"),
                                            ((96, 128, 192), "fp64"), ((128, 96, 192), "fp64"),
                                            ((128, 128, 256), "fp64"), ((32, 512, 512), "fp32"),
                                            ((512, 32, 512), "fp32"), ((64, 256, 512), "fp32"),
                                            ((256, 96, 192), "fp32"), ((192, 128, 192), "fp32"),
                                            ((128, 192, 256), "fp32"), ((256, 64, 512), "fp32")])
def test_large_fields(grid, precision):
    import smaiso_quasi_b200 as q
    cells = int(np.prod(grid))
    assert cells * (8 if precision == "fp64" else 4) > 16 << 20
    a = np.random.default_rng(cells).standard_normal(grid)
    for plan in ("STx", "iSTx", "STy", "iSTy"):
        ref = qo.r2r3d(a, qo.PLAN_KINDS[plan])
        got = q.R2RPlan(*grid, plan, precision=precision).execute_host(a)
        assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < TOL[precision], plan
