"""Particles and walls with a coordinate that is not finite, in the module calls on caller-made tables.  What such a record
does to a sum follows from the sums' own terms (a neighbour is left out at distance 0 or beyond the support radius, and
NaN is neither), so that a kernel's idle lanes and its way of leaving terms out may not show."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RE = 1.0


def buffers(pkg, x, rows, walls=(), wall_rows=None):
    """Device buffers of particles at (x, 0.1, 0.2) and walls at (w, 0, 0) with normals (1, 0, 0), with the given rows."""
    n = len(x)
    wall_rows = wall_rows or [[] for _ in x]
    dev = pkg.buffers.StepBuffers(pkg.buffers.TorchAlloc("cuda"), n, len(walls), 1)
    put = dev.alloc.copy_
    put(dev.fluid["x"], np.asarray(x))
    put(dev.fluid["y"], np.full(n, 0.1))
    put(dev.fluid["z"], np.full(n, 0.2))
    if len(walls):
        put(dev.walls["x"], np.asarray(walls, dtype=np.float64))
        put(dev.walls["normal_x"], np.ones(len(walls)))
    for table, r in ((dev.fluid_neighbors, rows), (dev.wall_neighbors, wall_rows)):
        put(table["offsets"], np.cumsum([0] + [len(k) for k in r]).astype(np.int32))
        put(table["indices"], np.array([j for k in r for j in k] + [0], dtype=np.int32))
    p = pkg.abi.default_params()
    p.support_radius = p.grid.cell_size = RE
    return dev, p


@pytest.mark.parametrize("bad", [np.nan, np.inf], ids=["nan", "inf"])
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [3, 12289], ids=["parts", "threads"])
def test_moments_of_an_empty_row(pkg, device_api, bad, kind, n):
    # no neighbours, no terms: the regularisation alone (lambda, as the trace is 0), beside a particle that has neighbours
    x = np.zeros(n)
    x[1], x[2] = 0.25, bad
    dev, p = buffers(pkg, x, [[1], [0]] + [[] for _ in range(n - 2)])
    ctx = device_api.Context(0)
    try:
        ctx.prepare_moments(dev, p, [kind])
    finally:
        ctx.close()
    m = dev.moments[kind]
    size = pkg.abi.MOMENT_SIZE[kind]
    inverse = dev.alloc.to_numpy(m["inverse_matrices"])[2 * size * size:3 * size * size].reshape(size, size)
    assert dev.alloc.to_numpy(m["moment_trace"])[2] == 0.0 and dev.alloc.to_numpy(m["info"])[2] == 0
    assert np.allclose(inverse, np.eye(size) / p.lsmps_regularization, rtol=1e-15, atol=0.0)


@pytest.mark.parametrize("n", [3, 131073], ids=["lanes", "threads"])
def test_label_sums_beyond_the_radius(pkg, device_api, n):
    # particle 2 is infinitely far from the one neighbour of its row: no weight, no sum
    import torch

    x = np.zeros(n)
    x[1], x[2] = 0.25, np.inf
    dev, p = buffers(pkg, x, [[1], [0], [0]] + [[] for _ in range(n - 3)])
    names = [k for k, _ in pkg.abi.SurfaceDiagnostics._fields_]
    out = {k: torch.full((n,), 7, dtype=torch.int32 if "count" in k else torch.float64, device="cuda") for k in names}
    ctx = device_api.Context(0)
    try:
        ctx.classify_surface(dev, p, pkg.abi.SurfaceDiagnostics(*(out[k].data_ptr() for k in names)))
    finally:
        ctx.close()
    assert [float(out[k][2]) for k in ("number_density", "number_density_ratio", "anisotropy")] == [0.0, 0.0, 0.0]
    assert float(out["number_density"][0]) == float(out["number_density"][1]) > 0.0


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("n", [2, 2049], ids=["parts", "threads"])
def test_moments_beside_a_wall_at_nan(pkg, device_api, kind, n):
    # the matrix of a particle that lists such a wall is NaN (info: the first pivot is not positive); others are not
    rows = [[1], [0]] + [[] for _ in range(n - 2)]
    dev, p = buffers(pkg, [0.0, 0.25] + [0.0] * (n - 2), rows, [-0.25, np.nan], [[0, 1, 0], [0, 0]] + [[] for _ in range(n - 2)])
    ctx = device_api.Context(0)
    try:
        ctx.prepare_moments(dev, p, [kind])
    finally:
        ctx.close()
    m = dev.moments[kind]
    trace, info = dev.alloc.to_numpy(m["moment_trace"]), dev.alloc.to_numpy(m["info"])
    assert np.isnan(trace[0]) and info[0] != 0
    assert np.isfinite(trace[1:]).all() and info[1] == 0
