"""The two label kernels (csrc/surface.cu): sets of up to 131,072 particles take sixteen lanes to a particle, larger ones
one thread.  Both have to give the labels of the oracle, exactly, and both the same diagnostics: the same box classified
as a set of its own and within a set above the line (copies of it side by side, so that each copy's rows are its own)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def diagnostics(pkg, torch, n):
    names = [k for k, _ in pkg.abi.SurfaceDiagnostics._fields_]
    out = {k: torch.zeros(n, dtype=torch.int32 if "count" in k else torch.float64, device="cuda") for k in names}
    return out, pkg.abi.SurfaceDiagnostics(*(out[k].data_ptr() for k in names))


def classify(pkg, api, case):
    import torch

    b = api.device_buffers(case)
    ctx = api.Context(0)
    try:
        ctx.build_neighbor_lists(b, case.params)
        out, d = diagnostics(pkg, torch, case.n_fluid)
        ctx.classify_surface(b, case.params, d)
    finally:
        ctx.close()
    return b.numpy("fluid")["surface_type"], {k: v.cpu().numpy() for k, v in out.items()}


def copies(pkg, case, many):
    """`many` copies of a case, shifted along y by an exact multiple of the cell size, further apart than r_e."""
    h = case.params.grid.cell_size
    width = int(np.ceil((max(case.fluid["y"].max(), case.walls["y"].max()) -
                         min(case.fluid["y"].min(), case.walls["y"].min())) / h)) + 2
    sets = []
    for part in (case.fluid, case.walls):
        new = {k: np.tile(v, many) for k, v in part.items()}
        new["y"] = new["y"] + np.repeat(np.arange(many) * (width * h), len(part["y"]))
        sets.append(new)
    big = pkg.cases.Case("copies", case.l0, sets[0], sets[1], case.params)
    pkg.cases.derive_grid(case.params, [sets[0]["x"], sets[1]["x"]], [sets[0]["y"], sets[1]["y"]],
                          [sets[0]["z"], sets[1]["z"]])
    return big


@pytest.mark.parametrize("n", [1, 2, 5, 9], ids=lambda n: f"{n}^3")
def test_small_sets_match_the_oracle(pkg, device_api, oracle, n):
    from lsmps3d_b200 import buffers

    case = pkg.cases.lattice_box(n=n, l0=0.01)
    got, _ = classify(pkg, device_api, case)
    host = buffers.StepBuffers(buffers.NumpyAlloc(), case.n_fluid, case.n_wall, case.n_cells)
    host.load_case(case)
    oracle.build_neighbor_lists(host, case.params)
    oracle.classify_surface(host, case.params)
    assert np.array_equal(got, host.fluid["surface_type"])


def test_both_kernels_agree(pkg, device_api):
    # y and the shifts are multiples of 2^-20, so that a copy's differences are the original's, bit for bit
    case = pkg.cases.splash_scattered(nx=24, ny=8, nz=24, l0=2.0**-7)
    for part in (case.fluid, case.walls):
        for k in "xyz":
            part[k] = np.round(part[k] * 2.0**20) * 2.0**-20
    p = case.params
    p.support_radius = p.grid.cell_size = 3.125 * case.l0
    pkg.cases.derive_grid(p, [case.fluid["x"], case.walls["x"]], [case.fluid["y"], case.walls["y"]],
                          [case.fluid["z"], case.walls["z"]])
    small, sd = classify(pkg, device_api, case)
    many = 131072 // case.n_fluid + 1
    big = copies(pkg, case, many)
    assert case.n_fluid <= 131072 < big.n_fluid
    large, ld = classify(pkg, device_api, big)
    n = case.n_fluid
    assert {1, 2, 3} <= set(np.unique(small).tolist())
    order = ("fluid_neighbor_count", "wall_neighbor_count")
    for k in sd:
        assert np.array_equal(ld[k][:n], sd[k], equal_nan=True), k
        assert k not in order or np.array_equal(ld[k].reshape(many, n), np.tile(sd[k], (many, 1))), k
    assert np.array_equal(large[:n], small)
