"""The fused step where its tiles and lane placements change: every supported
length on each axis, with the fewest rows and columns a grid may have, against
the oracle; and the transform forms (one launch up to 4 MB, separate passes
above, data that is not 16-byte aligned).

Tolerances: 1e-12 per quantity before the switches and 1e-11 behind them, those
of the step tests.  Behind them divv is (rho - rho_old)/dt over rho, and v takes
it up: their errors are those of rho over dt, 1e-14 / 1e-3 against values that
differ from grid to grid, and are left to the step tests.
"""
import numpy as np
import pytest

from oracle import quasi_oracle as qo

pytestmark = pytest.mark.gpu

GRIDS = [(8, 16, 16), (16, 8, 32), (32, 96, 64), (96, 32, 16), (192, 16, 96), (16, 192, 128), (128, 64, 16),
         (64, 128, 192), (256, 8, 32), (8, 256, 16), (512, 8, 16), (8, 512, 16), (8, 8, 512), (16, 32, 256)]


def rel(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(a - b) / n if n else np.linalg.norm(a)


def pair(variant, grid, ranks, precision, switch=1, ic="undulated"):
    import smaiso_quasi_b200 as q
    cfg = q.default_config(variant, *grid, emulate_ranks=ranks, precision=precision, divv_switch=switch)
    kw = dict(nx=grid[0], ny=grid[1], nz=grid[2], emulate_ranks=ranks, divv_switch=switch)
    o = qo.QuasiOracle(qo.Model(**kw) if variant == "quasi" else qo.Model.stb(**kw))
    psi0 = qo.ic_field(o.m, ic, seed=sum(grid))
    s = q.Simulation(cfg)
    s.set_psi(psi0)
    s.init()
    o.set_psi(psi0)
    o.init()
    return s, o


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("variant,ranks", [("quasi", 1), ("quasi", 4), ("stb", 2)])
def test_step_behind_the_switches_on_every_length(grid, variant, ranks):
    s, o = pair(variant, grid, ranks, "fp64", switch=1)
    for _ in range(4):   # the switches are at 1 and 2
        o.step()
    s.step(4)
    fields = ["psi", "psiq", "rho"] + (["p", "df"] if variant == "quasi" else ["dtpsi"])
    errs = {f: rel(s.field(f), o.field(f)) for f in fields}
    assert all(e < 1e-11 for e in errs.values()), errs


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("ranks", [1, 2])
def test_velocity_on_every_length(grid, ranks):
    s, o = pair("quasi", grid, ranks, "fp64", switch=200, ic="planar")
    for _ in range(3):
        o.step()
    s.step(3)
    errs = {f: rel(s.field(f), o.field(f)) for f in ("psi", "rho", "p")}
    errs["v"] = rel(np.stack([s.field(f) for f in ("vx", "vy", "vz")]), np.stack([o.field(f) for f in ("vx", "vy", "vz")]))
    assert all(e < 1e-12 for e in errs.values()), errs


@pytest.mark.parametrize("grid", GRIDS)
def test_fp32_step_on_every_length(grid):
    """FP32 against FP64, 10 steps: 1e-5, the form's bound, in psi and rho."""
    a, _ = pair("quasi", grid, 2, "fp32")
    b, _ = pair("quasi", grid, 2, "fp64")
    a.step(10)
    b.step(10)
    for f in ("psi", "rho"):
        assert rel(a.field(f), b.field(f)) < 1e-5, f


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_checkpoint_resumes_the_same_step(tmp_path, precision):
    """Between steps the state holds spectra that the file does not: they are
    derived when it is loaded, bit for bit."""
    a, _ = pair("quasi", (32, 16, 64), 2, precision)
    a.step(5)
    a.save(tmp_path / "c.bin")
    b, _ = pair("quasi", (32, 16, 64), 2, precision)
    b.step(2)
    b.load(tmp_path / "c.bin")
    a.step(6)
    b.step(6)
    for f in ("psi", "rho", "vx", "vz", "p", "divv"):
        assert np.array_equal(a.field(f), b.field(f)), f


@pytest.mark.parametrize("grid", [(64, 64, 128), (64, 128, 128), (256, 16, 256), (256, 8, 256), (8, 256, 256), (128, 128, 128),
                                  (16, 16, 512)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-14), ("fp32", 2e-6)])
def test_transform_forms(grid, precision, tol):
    """On both sides of the one-launch form's size, on aligned data and on data one
    pair of floats or one value off."""
    import torch

    import smaiso_quasi_b200 as q
    dt = torch.float64 if precision == "fp64" else torch.float32
    a = np.random.default_rng(3).standard_normal(grid)
    for plan in ("STy", "iSTx"):
        ref = qo.r2r3d(a, qo.PLAN_KINDS[plan])
        p = q.R2RPlan(*grid, plan, precision=precision)
        for off in (0, 2, 1) if precision == "fp32" else (0, 1):
            buf = torch.empty(a.size + off, dtype=dt, device="cuda")
            x = buf[off:]
            x.copy_(torch.from_numpy(a.astype(np.float64 if precision == "fp64" else np.float32)).reshape(-1))
            torch.cuda.synchronize()
            p.execute_device(x.data_ptr())
            assert rel(x.double().cpu().numpy().reshape(grid), ref) < tol, (plan, off)
