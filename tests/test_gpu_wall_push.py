"""The update and anti-penetration stage of the pressure correction (csrc/correction.cu) on both sides of its line (131,072
particles: below, eight lanes walk a particle's walls; above, its own thread): one particle, sets that end inside a block,
and a set repeated past the line, with a clearance at which most walls push, against the reference's loop in numpy.
Positions and velocities (smoothing off) within 200 roundings of their scale: a row has at most 100 walls here, each adding
a few roundings to a state whose size it does not raise."""

import numpy as np
import pytest

from test_gpu_moment_parts import repeated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,copies", [(1, 1), (17, 1), (2000, 1), (2000, 66)])
def test_push(pkg, device_api, oracle, n, copies):
    case = pkg.cases.CASES["dam_break_shuffled"](nx=20, ny=10, nz=20, l0=0.005)
    host = pkg.buffers.StepBuffers(pkg.buffers.NumpyAlloc(), case.n_fluid, case.n_wall, case.n_cells)
    host.load_case(case)
    p = case.params
    oracle.build_neighbor_lists(host, p)
    p.wall_clearance_ratio, p.velocity_smoothing_strength = 1.2, 0.0
    clearance = p.wall_clearance_ratio * p.particle_spacing
    dev = repeated(pkg, host, n, copies)
    rng = np.random.default_rng(n)
    v0, vt = rng.standard_normal((2, n, 3))
    put, get = dev.alloc.copy_, dev.alloc.to_numpy
    for k, c in enumerate(("vx", "vy", "vz")):
        put(dev.fluid[c], np.tile(v0[:, k], copies))
        put(dev.temporary_velocity[c], np.tile(vt[:, k], copies))
    put(dev.fluid["pressure"], np.tile(100.0 * rng.random(n), copies))
    x0 = np.stack([host.fluid[c][:n] for c in "xyz"], 1)
    ctx = device_api.Context(0)
    try:
        ctx.prepare_moments(dev, p, [1])
        ctx.pressure_correction(dev, p)
    finally:
        ctx.close()
    g, s = (np.stack([get(f[c])[:n] for c in "xyz"], 1) for f in (dev.pressure_gradient, dev.ps_displacement))
    wo, wi = dev.csr_rows("wall")
    wall, normal = (np.stack([host.walls[c] for c in names], 1)
                    for names in (("x", "y", "z"), ("normal_x", "normal_y", "normal_z")))
    v = vt - p.time_step / p.density * g
    x = x0 + 0.5 * p.time_step * (v0 + v) + s
    pushes = 0
    for i in range(n):
        for j in wi[wo[i]:wo[i + 1]]:
            sd = np.dot(x[i] - wall[j], normal[j])
            if sd >= clearance:
                continue
            x[i] += (clearance - sd) * normal[j]
            nv = np.dot(v[i], normal[j])
            if nv < 0.0:
                v[i] -= nv * normal[j]
            pushes += 1
    assert pushes > n // 4 or n == 1
    for c in range(copies):
        at = slice(c * n, (c + 1) * n)
        for k, (a, b) in enumerate((("x", "vx"), ("y", "vy"), ("z", "vz"))):
            assert np.max(np.abs(get(dev.fluid[a])[at] - x[:, k])) <= 200 * 2.0**-52 * max(1.0, np.abs(x).max())
            assert np.max(np.abs(get(dev.fluid[b])[at] - v[:, k])) <= 200 * 2.0**-52 * max(1.0, np.abs(v).max())
