"""The neighbour tables' block passes (csrc/neighbors.cu) at their edges: home cells of 1, 32, 33 and 65 particles (one
round of lanes, one more, three), rows of up to 324 and 325 entries (listed in two and three pieces of 162), 1,024 and
1,025 candidates (staged, and tested from global memory), empty cells between the occupied ones, and a capacity that
ends inside a row.  The host oracle's tables have to be the same to the entry."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# particles (fluid, wall) in cells of a 5 x 4 x 3 grid, by cell coordinates
CASES = {
    "lanes": ({(0, 0, 0): 1, (1, 1, 1): 32, (2, 1, 1): 33, (4, 3, 2): 65, (0, 3, 1): 2}, {(1, 1, 0): 33, (3, 3, 2): 1}),
    "two-pieces": ({(1, 1, 1): 325, (4, 0, 0): 5}, {(2, 2, 2): 324}),
    "three-pieces": ({(1, 1, 1): 300, (2, 1, 1): 26, (3, 1, 1): 7}, {(2, 2, 2): 400}),
    "staged": ({(1, 1, 1): 1000, (2, 2, 2): 24, (4, 2, 2): 9}, {(0, 0, 0): 1024}),
    "over": ({(1, 1, 1): 1000, (2, 2, 2): 25, (4, 2, 2): 9}, {(0, 0, 0): 1025}),
}


@pytest.mark.parametrize("cut", [0, 40], ids=["whole", "cut"])
@pytest.mark.parametrize("name", CASES)
def test_tables(pkg, device_api, oracle, name, cut):
    dims = (5, 4, 3)
    rng = np.random.default_rng(len(name))
    p = pkg.cases.hydrostatic_box(n=4, l0=0.01).params
    h = p.support_radius
    p.grid.cell_size = h
    p.grid.origin[:] = (-0.3, 0.1, 0.7)
    p.grid.dims[:] = dims

    def points(cells):
        at = np.concatenate([np.repeat([c], k, 0) for c, k in cells.items()]) + rng.uniform(0.01, 0.99, (sum(cells.values()), 3))
        return rng.permutation(np.array(p.grid.origin[:]) + h * at)

    fluid, wall = points(CASES[name][0]), points(CASES[name][1])
    bufs = [pkg.buffers.StepBuffers(a, len(fluid), len(wall), 60, 1100, 1100)
            for a in (pkg.buffers.NumpyAlloc(), pkg.buffers.TorchAlloc("cuda"))]
    for b in bufs:
        for k, axis in enumerate("xyz"):
            b.alloc.copy_(b.fluid[axis], fluid[:, k])
            b.alloc.copy_(b.walls[axis], wall[:, k])
    host, dev = bufs
    oracle.build_neighbor_lists(host, p)
    ctx = device_api.Context(0)
    try:
        if not cut:
            ctx.build_neighbor_lists(dev, p)
        else:
            want = int(host.fluid_neighbors["offsets"][-1])
            dev.alloc.copy_(dev.fluid_neighbors["indices"], np.full(want, -7, np.int32))
            dev.cap_f = want - cut
            with pytest.raises(device_api.LsmpsError) as e:
                ctx.build_neighbor_lists(dev, p)
            assert e.value.status == pkg.abi.CAPACITY_EXCEEDED and ctx.required == want
    finally:
        ctx.close()
    for which in ("fluid", "wall"):
        table = getattr(dev, which + "_neighbors")
        go, gi = (dev.alloc.to_numpy(table[k]) for k in ("offsets", "indices"))
        ho, hi = host.csr_rows(which)
        assert np.array_equal(go, ho)
        n = int(ho[-1])
        end = n - cut if which == "fluid" else n
        assert np.array_equal(gi[:end], hi[:end])
        assert np.all(gi[end:n] == -7)
