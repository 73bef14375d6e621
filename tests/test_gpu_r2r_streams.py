"""r2r plans as a program with several streams, threads and graphs uses them."""
import threading

import numpy as np
import pytest

from oracle import quasi_oracle as qo

pytestmark = pytest.mark.gpu

# column passes without tensor copies up to 16 MB; the last is above in FP64
GRIDS = [(16, 16, 32), (64, 64, 128), (96, 96, 192), (128, 128, 256)]
TOL = {"fp64": 1e-14, "fp32": 2e-6}


def case(grid, precision, seed):
    import torch
    a = np.random.default_rng(seed).standard_normal(grid)
    x = torch.from_numpy(a).to("cuda", torch.float64 if precision == "fp64" else torch.float32)
    return a, x


def err(x, a, plan):
    ref = qo.r2r3d(a, qo.PLAN_KINDS[plan])
    return np.linalg.norm(x.double().cpu().numpy() - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_inside_a_stream_capture(grid, precision):
    import torch

    import smaiso_quasi_b200 as q
    a, x = case(grid, precision, 1)
    work = torch.empty_like(x)
    p = q.R2RPlan(*grid, "STx", precision=precision)
    graph, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=st):
        work.copy_(x)
        p.execute_device(work.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert err(work, a, "STx") < TOL[precision]
    del graph


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("threads", [False, True])
def test_beside_other_streams(grid, threads):
    """Four plans on four streams, from one host thread or four, beside matrix
    products on a fifth."""
    import torch

    import smaiso_quasi_b200 as q
    plans = ["CT", "iSTz", "STy", "iCT"]
    made = [case(grid, "fp64", s) for s in range(4)]
    ps = [q.R2RPlan(*grid, plan) for plan in plans]
    streams = [torch.cuda.Stream() for _ in range(5)]
    work = [torch.empty_like(x) for _, x in made]
    m = torch.randn(2048, 2048, device="cuda")
    torch.cuda.synchronize()

    def passes(k):
        with torch.cuda.stream(streams[k]):
            for _ in range(20):
                work[k].copy_(made[k][1])
                ps[k].execute_device(work[k].data_ptr(), streams[k].cuda_stream)

    with torch.cuda.stream(streams[4]):
        for _ in range(20):
            m = (m @ m).clamp(-1, 1)
    if threads:
        ts = [threading.Thread(target=passes, args=(k,)) for k in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for k in range(4):
            passes(k)
    torch.cuda.synchronize()
    for k in range(4):
        assert err(work[k], made[k][0], plans[k]) < TOL["fp64"], k


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("grid", [(64, 64, 64), (64, 64, 128), (16, 256, 64), (128, 128, 64)])
def test_needs_no_idle_gpu(grid, precision):
    """A transform ends while a kernel of another stream still holds a part of one
    SM: its CTAs need not be resident all at once."""
    import torch

    import smaiso_quasi_b200 as q
    a, x = case(grid, precision, 2)
    p = q.R2RPlan(*grid, "CT", precision=precision)
    other, st = torch.cuda.Stream(), torch.cuda.Stream()
    work = torch.zeros_like(x)
    p.execute_device(work.data_ptr(), st.cuda_stream)   # loaded
    work.copy_(x)
    torch.cuda.synchronize()
    held, done = torch.cuda.Event(), torch.cuda.Event()
    with torch.cuda.stream(other):
        torch.cuda._sleep(1_000_000_000)   # half a second
        held.record()
    p.execute_device(work.data_ptr(), st.cuda_stream)
    done.record(st)
    done.synchronize()
    assert not held.query()
    torch.cuda.synchronize()
    assert err(work, a, "CT") < TOL[precision]
