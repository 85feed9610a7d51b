"""The counting sort behind the cell lists (csrc/cells.cu) at its edges: cells of one, 32, 33, 1,024 and 1,025 particles
and all particles in one cell (ordered by shuffles, by comparison, by a walk over the set), cell counts on both sides of
the one-block scan (8,192) and of its tiles, one particle and none; against numpy's stable sort of the cell ids."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(pkg, device_api, ids, dims):
    """build_cell_list of particles placed at the centres of the cells `ids`."""
    import torch

    abi = pkg.abi
    n, ncell = len(ids), int(np.prod(dims))
    g = abi.Grid()
    g.cell_size = 0.5
    g.origin[:] = (-1.0, 2.0, 0.25)
    g.dims[:] = dims
    at = np.stack([ids % dims[0], ids // dims[0] % dims[1], ids // (dims[0] * dims[1])], 1)
    xyz = [torch.from_numpy(g.origin[k] + 0.5 * (at[:, k] + 0.5)).cuda() for k in range(3)]
    t = {k: torch.full((max(m, 1),), -9, dtype=torch.int32, device="cuda")
         for k, m in (("cell_ids", n), ("sorted_indices", n), ("cell_begin", ncell), ("cell_end", ncell))}
    c = abi.Cells()
    c.particle_count, c.cell_count = n, ncell
    for k, v in t.items():
        setattr(c, k, v.data_ptr())
    ctx = device_api.Context(0)
    try:
        ctx.build_cell_list(*(v.data_ptr() if n else None for v in xyz), n, g, c)
    finally:
        ctx.close()
    return {k: v.cpu().numpy()[: n if "cell_b" not in k and "cell_e" not in k else ncell] for k, v in t.items()}


def check(got, ids, ncell):
    order = np.argsort(ids, kind="stable")
    assert np.array_equal(got["sorted_indices"], order)
    assert np.array_equal(got["cell_ids"], ids[order])
    count = np.bincount(ids, minlength=ncell)
    end = np.cumsum(count)
    assert np.array_equal(got["cell_begin"], np.where(count > 0, end - count, -1))
    assert np.array_equal(got["cell_end"], np.where(count > 0, end, -1))


@pytest.mark.parametrize("counts", [[1], [32, 33, 0, 31], [1024, 1025, 1], [5000], [0, 40, 2000, 0, 33, 1]],
                         ids=["one", "warp", "many", "all-in-one", "mixed"])
@pytest.mark.parametrize("dims", [(3, 2, 1), (32, 16, 16), (33, 17, 17)], ids=["6", "8192", "9537"])
def test_cells(pkg, device_api, counts, dims):
    ncell = int(np.prod(dims))
    rng = np.random.default_rng(sum(counts) + ncell)
    cells = rng.permutation(ncell)[: len(counts)]
    ids = rng.permutation(np.repeat(cells, counts))
    check(build(pkg, device_api, ids, dims), ids, ncell)


@pytest.mark.parametrize("n", [0, 1, 2047, 2049, 300000])
def test_counts(pkg, device_api, n):
    dims = (40, 41, 43)
    ids = np.random.default_rng(n).integers(0, int(np.prod(dims)), n)
    check(build(pkg, device_api, ids, dims), ids, int(np.prod(dims)))
