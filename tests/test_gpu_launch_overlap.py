"""Kernels are launched with their blocks allowed onto the GPU before the kernel before them has ended, where they wait
for it (csrc/common.cuh).  With profiling on, an event stands between every two launches, so none is early, and under
capture none is asked for: the states and solutions of all three have to be the same, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "vx", "vy", "vz", "pressure", "surface_type")


def steps(pkg, api, form, how, count):
    import torch

    case = pkg.cases.CASES["dam_break_shuffled"](nx=12, ny=8, nz=12, l0=0.005)
    dev = api.device_buffers(case)
    stream = torch.cuda.Stream()
    ctx = api.Context(0, precision=getattr(pkg.abi, "PRECISION_" + form))
    try:
        ctx.build_neighbor_lists(dev, case.params)
        ctx.classify_surface(dev, case.params)
        state = dev.step_state(case.params)
        ctx.reserve(dev.n_fluid, dev.n_wall, dev.n_cells)
        ctx.set_synchronous(False)
        torch.cuda.synchronize()
        ctx.set_stream(stream.cuda_stream)
        ctx.set_profiling(how == "events")
        if how == "graph":
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                ctx.step(dev, case.params, state)
            with torch.cuda.stream(stream):
                for _ in range(count):
                    g.replay()
        else:
            for _ in range(count):
                ctx.step(dev, case.params, state)
        ctx.synchronize()
        torch.cuda.synchronize()
        return dev.numpy("fluid"), dev.csr_rows("fluid")
    finally:
        ctx.close()


@pytest.mark.parametrize("form", ["PLAIN", "MIXED"])
def test_steps(pkg, device_api, form):
    want, rows = steps(pkg, device_api, form, "events", 40)
    for how in ("early", "graph"):
        got, r = steps(pkg, device_api, form, how, 40)
        for k in FIELDS:
            assert np.array_equal(got[k], want[k]), (how, k)
        assert np.array_equal(r[0], rows[0]) and np.array_equal(r[1], rows[1]), how


@pytest.mark.parametrize("n", [1, 300, 8000, 110000])
def test_solve(pkg, device_api, n):
    import torch

    rng = np.random.default_rng(n)
    ro = (np.arange(n + 1) * 5).astype(np.int32)
    ci = rng.integers(0, n, 5 * n).astype(np.int32)
    ci[ro[:-1]] = np.arange(n)
    va = rng.standard_normal(5 * n)
    va[ro[:-1]] += 6.0
    t = [torch.as_tensor(a).cuda() for a in (ro, ci, va, rng.standard_normal(n))]
    m = pkg.abi.CsrMatrix(n, n, 5 * n, *(a.data_ptr() for a in t[:3]))
    o = pkg.abi.default_solver_options()
    o.max_iters, o.tolerance, o.clamp_negative = 70, 1e-10, 0
    got = []
    for profiling in (True, False):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        ctx = device_api.Context(0)
        try:
            ctx.set_profiling(profiling)
            rep = ctx.solve_csr(m, t[3].data_ptr(), x.data_ptr(), o)
        finally:
            ctx.close()
        got.append((x.cpu().numpy(), rep.iterations, rep.final_residual))
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1:] == got[1][1:]
