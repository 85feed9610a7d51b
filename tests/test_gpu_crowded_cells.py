"""Cell lists of crowded cells (csrc/cells.cu): the places of a cell's particles are found by comparison, those of a cell
with more than 1,024 particles and a 32nd of its set by a walk over the set, and a set of more than 128 particles a
cell on average is sorted.  Their results against numpy's stable sort and the oracle's tables at the edges of those
rules, and their times against that of the same number of particles spread evenly."""

import numpy as np
import pytest

from test_gpu_cell_sort import build, check

pytestmark = pytest.mark.gpu


def crowd(n, ncell, many, seed=0):
    """Cell ids of n particles, `many` of them in cell 5 and the others anywhere else."""
    rng = np.random.default_rng(n + many + seed)
    ids = rng.integers(0, ncell - 1, n)
    ids += ids >= 5
    ids[rng.permutation(n)[:many]] = 5
    return ids


@pytest.mark.parametrize("n,many", [(40001, 1250), (40001, 1251), (40001, 30000), (9000, 1024), (9000, 1025), (3001, 3001)])
def test_one_crowded_cell(pkg, device_api, n, many):
    dims = (31, 20, 13)
    ids = crowd(n, int(np.prod(dims)), many)
    check(build(pkg, device_api, ids, dims), ids, int(np.prod(dims)))


@pytest.mark.parametrize("dims", [(3, 2, 1), (17, 17, 1)], ids=["6", "289"])
@pytest.mark.parametrize("extra", [0, 1, 5000])
def test_many_per_cell(pkg, device_api, dims, extra):
    ncell = int(np.prod(dims))
    ids = np.random.default_rng(ncell + extra).integers(0, ncell, 128 * ncell + extra)
    check(build(pkg, device_api, ids, dims), ids, ncell)


@pytest.mark.parametrize("dims,n_fluid,n_wall,at", [((2, 1, 1), 101, 3000, None), ((2, 1, 1), 900, 50, None),
                                                   ((2, 1, 1), 900, 3000, None), ((30, 10, 10), 101, 1500, 0.1),
                                                   ((30, 10, 10), 1500, 77, 0.1)],
                         ids=["walls-sorted", "fluid-sorted", "both-sorted", "walls-walked", "fluid-walked"])
def test_tables(pkg, device_api, oracle, dims, n_fluid, n_wall, at):
    """Fluid and walls anywhere in the grid, or within `at` of one point."""
    rng = np.random.default_rng(n_fluid + n_wall)
    p = pkg.abi.default_params()
    p.support_radius, p.grid.cell_size = 0.2, 1.0
    p.grid.dims[:] = dims
    p.grid.origin[:] = (0.0, 0.0, 0.0)
    size = np.asarray(dims) if at is None else np.full(3, at)
    got = []
    points = [size * rng.random((n, 3)) + (0.0 if at is None else 0.3) for n in (n_fluid, n_wall)]
    for alloc in (pkg.buffers.NumpyAlloc(), pkg.buffers.TorchAlloc("cuda")):
        b = pkg.buffers.StepBuffers(alloc, n_fluid, n_wall, int(np.prod(dims)), 1500, 1500)
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
        got.append([*b.csr_rows("fluid"), *b.csr_rows("wall"), *b.numpy("fluid_cells").values(), *b.numpy("wall_cells").values()])
    assert got[0][0][-1] > 0 and got[0][2][-1] > 0
    for want, have in zip(*got):
        assert np.array_equal(want, have)


def best_time(pkg, device_api, ids, dims):
    """Shortest of a few builds, us."""
    import torch

    times = []

    def timed(ctx_build):
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx_build()
            b.record()
            torch.cuda.synchronize()
            times.append(1e3 * a.elapsed_time(b))

    class Api:
        class Context(device_api.Context):
            def build_cell_list(self, *args):
                timed(lambda: device_api.Context.build_cell_list(self, *args))

    build(pkg, Api, ids, dims)
    return min(times)


def test_time_does_not_follow_the_crowd(pkg, device_api):
    """300,000 particles: at most four times as long as evenly spread (about 35 us) with 1,025 or 9,000 of them in one cell,
    or with 37,500 in each (about 40, 150 and 30; ordered by one warp's walk per cell 2,300 to 2,900; a walk costs half a
    nanosecond a particle, hence the wider line for the cell that is walked)."""
    n, fine = 300000, (22, 22, 22)
    even = best_time(pkg, device_api, np.random.default_rng(1).integers(0, 22**3, n), fine)
    assert best_time(pkg, device_api, crowd(n, 22**3, 1025), fine) < 4 * even
    assert best_time(pkg, device_api, np.random.default_rng(2).integers(0, 8, n), (2, 2, 2)) < 4 * even
    assert best_time(pkg, device_api, crowd(n, 22**3, 9000), fine) < 12 * even
    assert best_time(pkg, device_api, crowd(n, 22**3, 200000), fine) < 24 * even
