"""Moment sums in parts (csrc/moment.cu: small sets, a block to 32 particles) against the sums of a thread per particle,
which larger sets take: a set on one side of a line (12,288 particles for the sums, 2,048 for the wall terms) and the same
set repeated until it is past both, whose first copy's matrices have to be the same, bit for bit.  One particle, sets that
end inside a block, the last and first sizes around the wall terms' line; all four kinds together and each alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("inverse_matrices", "moment_trace", "regularization_added", "info")


def repeated(pkg, host, n, copies):
    """Device buffers of the first n particles of `host` (rows cut to entries below n), `copies` times over."""
    def rows(table, keep):
        o, i = host.csr_rows(table)
        o, i = o[: n + 1], i[: o[n]]
        counts = np.diff(o)
        ok = keep(i)
        row = np.repeat(np.arange(n), counts)[ok]
        return np.bincount(row, minlength=n), i[ok]

    fc, fi = rows("fluid", lambda i: i < n)
    wc, wi = rows("wall", lambda i: i >= 0)
    dev = pkg.buffers.StepBuffers(pkg.buffers.TorchAlloc("cuda"), n * copies, host.n_wall, host.n_cells,
                                  fluid_capacity=max(1, copies * len(fi)), wall_capacity=max(1, copies * len(wi)))
    put = dev.alloc.copy_
    for k in "xyz":
        put(dev.fluid[k], np.tile(host.fluid[k][:n], copies))
    for k in dev.walls:
        put(dev.walls[k], host.walls[k])
    put(dev.fluid_neighbors["offsets"], np.concatenate([[0], np.cumsum(np.tile(fc, copies))]).astype(np.int32))
    put(dev.fluid_neighbors["indices"], (np.tile(fi, copies) + n * np.repeat(np.arange(copies), len(fi))).astype(np.int32))
    put(dev.wall_neighbors["offsets"], np.concatenate([[0], np.cumsum(np.tile(wc, copies))]).astype(np.int32))
    put(dev.wall_neighbors["indices"], np.tile(wi, copies).astype(np.int32))
    return dev


def moments(pkg, ctx, host, params, n, copies, kinds):
    dev = repeated(pkg, host, n, copies)
    ctx.prepare_moments(dev, params, kinds)
    return {k: {f: dev.alloc.to_numpy(dev.moments[k][f]) for f in KEYS} for k in kinds}


@pytest.mark.parametrize("kinds", [[0, 1, 2, 3], [0], [1], [2], [3]], ids=["all", "0", "1", "2", "3"])
@pytest.mark.parametrize("n", [1, 31, 33, 2048, 2049, 3000])
def test_same_bits(pkg, device_api, oracle, n, kinds):
    case = pkg.cases.CASES["dam_break_shuffled"](nx=20, ny=10, nz=20, l0=0.005)
    host = pkg.buffers.StepBuffers(pkg.buffers.NumpyAlloc(), case.n_fluid, case.n_wall, case.n_cells)
    host.load_case(case)
    oracle.build_neighbor_lists(host, case.params)
    ctx = device_api.Context(0)
    try:
        small = moments(pkg, ctx, host, case.params, n, 1, kinds)
        large = moments(pkg, ctx, host, case.params, n, 12288 // n + 2, kinds)
    finally:
        ctx.close()
    for k in kinds:
        m2 = len(small[k]["inverse_matrices"]) // n
        for f in KEYS:
            per = m2 if f == "inverse_matrices" else 1
            assert np.array_equal(small[k][f], large[k][f][: n * per], equal_nan=True), (k, f)
        assert np.any(small[k]["moment_trace"] != 0.0) or n == 1
