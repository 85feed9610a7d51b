"""Sizes at which the solve's kernels change (csrc/solve.cu): basis widths of 8, 16, 24 and up to 64 vectors, one product
kernel with the dot products and one without (100,000 rows), rows of no, one and many entries, a single row; against the
oracle's GMRES (same algorithm, other orders of summation) with the iteration counts equal, and residuals recomputed."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n, per_row, seed, dominant):
    """Random rows (row 0 has its diagonal only), columns unsorted, diagonal first as in the PPE's layout."""
    rng = np.random.default_rng(seed)
    counts = rng.integers(0, 2 * per_row + 1, n)
    counts[0] = 0
    ro = np.concatenate([[0], np.cumsum(counts + 1)]).astype(np.int32)
    ci = rng.integers(0, n, ro[-1]).astype(np.int32)
    va = rng.standard_normal(ro[-1])
    ci[ro[:-1]] = np.arange(n)
    va[ro[:-1]] = dominant * np.sqrt(counts + 1.0) * np.where(rng.random(n) < 0.5, 1.0, 1.5)
    return ro, ci, va, rng.standard_normal(n)


def residual(ro, ci, va, b, x):
    rows = np.repeat(np.arange(len(b)), np.diff(ro))
    return np.linalg.norm(b - np.bincount(rows, weights=va * x[ci], minlength=len(b)))


def solve(pkg, device_api, ro, ci, va, b, **kw):
    import torch

    o = pkg.abi.default_solver_options()
    for k, v in kw.items():
        setattr(o, k, v)
    t = [torch.as_tensor(a).cuda() for a in (ro, ci, va, b)]
    x = torch.full((len(b),), 7.0, dtype=torch.float64, device="cuda")
    m = pkg.abi.CsrMatrix(len(b), len(b), len(va), *(a.data_ptr() for a in t[:3]))
    ctx = device_api.Context(0)
    try:
        rep = ctx.solve_csr(m, t[3].data_ptr(), x.data_ptr(), o)
    finally:
        ctx.close()
    return x.cpu().numpy(), rep


@pytest.mark.parametrize("n,restart", [(1, 1), (3, 2), (257, 7), (257, 8), (1000, 9), (1000, 17), (2000, 25), (2000, 64)])
def test_widths(pkg, device_api, oracle, n, restart):
    ro, ci, va, b = system(n, 6, 10 * n + restart, 1.3)
    kw = dict(restart=restart, max_iters=150, tolerance=1e-9, clamp_negative=0)
    x, rep = solve(pkg, device_api, ro, ci, va, b, **kw)
    o = pkg.abi.default_solver_options()
    for k, v in kw.items():
        setattr(o, k, v)
    want = np.zeros(n)
    st, ref = oracle.solve_ppe(ro, ci, va, b, want, o)
    assert st == 0
    assert rep.iterations == ref.iterations and rep.converged == ref.converged
    # both residuals are those of their own iterates; the iterates agree to the rounding of a converged solve
    assert abs(rep.final_residual - residual(ro, ci, va, b, x)) <= 1e-12 * np.linalg.norm(b)
    assert np.max(np.abs(x - want)) <= 1e-7 * np.max(np.abs(want))


@pytest.mark.parametrize("n", [100000, 100001], ids=["fused", "apart"])
def test_product_line(pkg, device_api, n):
    ro, ci, va, b = system(n, 5, n, 4.0)
    x, rep = solve(pkg, device_api, ro, ci, va, b, tolerance=1e-10, clamp_negative=0)
    assert rep.converged == 1
    assert residual(ro, ci, va, b, x) <= 1.01e-10 * np.linalg.norm(b)
    again, rep2 = solve(pkg, device_api, ro, ci, va, b, tolerance=1e-10, clamp_negative=0)
    assert np.array_equal(x, again) and rep2.iterations == rep.iterations


def test_no_iterations_and_converged_start(pkg, device_api):
    ro, ci, va, b = system(500, 5, 3, 4.0)
    x, rep = solve(pkg, device_api, ro, ci, va, b, max_iters=0)
    assert rep.iterations == 0 and rep.converged == 0 and not x.any()
    x, rep = solve(pkg, device_api, ro, ci, va, np.zeros_like(b))
    assert rep.iterations == 0 and rep.converged == 1 and not x.any()
