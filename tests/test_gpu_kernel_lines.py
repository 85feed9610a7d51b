"""Edges that the tests of single kernels leave out: neighbour rows of as many entries as csrc/neighbors.cu lists at a time
(162) and one more, once, twice and three times; moment sums at the last size that is summed in parts (12,288) and the first
that is not; steps of a set large enough for the kernels of large sets, launched early and one after the other."""

import numpy as np
import pytest

import test_gpu_moment_parts as parts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries", [161, 162, 163, 324, 325, 487])
def test_row_lengths(pkg, device_api, oracle, entries):
    n = entries + 1  # every particle lists all others, and every wall
    rng = np.random.default_rng(n)
    points = [1.0 + 0.2 * rng.random((m, 3)) for m in (n, entries)]
    p = pkg.abi.default_params()
    p.support_radius, p.grid.cell_size = 0.4, 0.41
    p.grid.dims[:] = (5, 6, 7)
    p.grid.origin[:] = (0.0, 0.0, 0.0)
    got = []
    for alloc in (pkg.buffers.NumpyAlloc(), pkg.buffers.TorchAlloc("cuda")):
        b = pkg.buffers.StepBuffers(alloc, n, entries, 210, entries, entries)
        for group, x in zip((b.fluid, b.walls), points):
            for c, k in enumerate("xyz"):
                alloc.copy_(group[k], x[:, c].copy())
        if alloc.device == "cpu":
            oracle.build_neighbor_lists(b, p)
        else:
            ctx = device_api.Context(0)
            try:
                ctx.build_neighbor_lists(b, p)
            finally:
                ctx.close()
        got.append([*b.csr_rows("fluid"), *b.csr_rows("wall")])
    assert np.all(np.diff(got[0][0]) == entries) and np.all(np.diff(got[0][2]) == entries)
    for want, have in zip(*got):
        assert np.array_equal(want, have)


@pytest.mark.parametrize("n", [12288, 12289])
def test_moment_line(pkg, device_api, oracle, n):
    case = pkg.cases.CASES["dam_break_shuffled"](nx=32, ny=16, nz=25, l0=0.005)
    host = pkg.buffers.StepBuffers(pkg.buffers.NumpyAlloc(), case.n_fluid, case.n_wall, case.n_cells)
    host.load_case(case)
    oracle.build_neighbor_lists(host, case.params)
    ctx = device_api.Context(0)
    kinds = [0, 1, 2]
    try:
        one = parts.moments(pkg, ctx, host, case.params, n, 1, kinds)
        two = parts.moments(pkg, ctx, host, case.params, n, 2, kinds)
    finally:
        ctx.close()
    for k in kinds:
        for f in parts.KEYS:
            for half in (0, 1):
                m = len(one[k][f])
                assert np.array_equal(one[k][f], two[k][f][half * m:(half + 1) * m], equal_nan=True), (k, f, half)


@pytest.mark.parametrize("form", ["PLAIN", "MIXED"])
def test_large_steps_launched_early(pkg, device_api, form):
    import torch

    case = pkg.cases.CASES["dam_break_shuffled"](nx=66, ny=32, nz=66, l0=0.005)
    assert case.n_fluid > 131072
    got = []
    for events in (True, False):  # an event between every two launches; none
        dev = device_api.device_buffers(case)
        ctx = device_api.Context(0, precision=getattr(pkg.abi, "PRECISION_" + form))
        try:
            ctx.build_neighbor_lists(dev, case.params)
            ctx.classify_surface(dev, case.params)
            state = dev.step_state(case.params)
            ctx.set_synchronous(False)
            ctx.set_profiling(events)
            for _ in range(6):
                ctx.step(dev, case.params, state)
            ctx.synchronize()
            torch.cuda.synchronize()
            total = int(dev.fluid_neighbors["offsets"][-1])
            got.append([dev.fluid[k].cpu().numpy() for k in ("x", "y", "z", "vx", "vy", "vz", "surface_type")]
                       + [dev.fluid_neighbors["indices"][:total].cpu().numpy(), dev.ppe["values"].cpu().numpy()])
        finally:
            ctx.close()
        del dev
    for a, b in zip(*got):
        assert np.array_equal(a, b)
