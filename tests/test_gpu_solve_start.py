"""Solves that have nothing, or little, to do (csrc/solve.cu): a system whose first residual meets the target, or with no
iterations allowed, queues no Arnoldi step (each is three launches or more, which return at once but are launched), and one
that converges in its first step few beyond it.  NaN in the matrix shows with a zero right-hand side too."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(pkg, n, bad=False):
    import torch

    rng = np.random.default_rng(n)
    ro = (np.arange(n + 1) * 5).astype(np.int32)
    ci = rng.integers(0, n, 5 * n).astype(np.int32)
    ci[ro[:-1]] = np.arange(n)
    va = 0.01 * rng.standard_normal(5 * n)
    va[ro[:-1]] += 2.0
    if bad:
        va[7] = np.nan
    t = [torch.as_tensor(a).cuda() for a in (ro, ci, va)]
    return t, pkg.abi.CsrMatrix(n, n, 5 * n, *(a.data_ptr() for a in t))


def solve(pkg, api, matrix, b, x, **options):
    o = pkg.abi.default_solver_options()
    o.restart, o.clamp_negative = 64, 0
    for k, v in options.items():
        setattr(o, k, v)
    ctx = api.Context(0)
    try:
        rep = ctx.solve_csr(matrix, b.data_ptr(), x.data_ptr(), o)
        return rep, ctx.launch_count
    finally:
        ctx.close()


@pytest.mark.parametrize("n", [1, 3000, 120000])
def test_nothing_to_do(pkg, device_api, n):
    import torch

    keep, m = system(pkg, n)
    b = torch.as_tensor(np.random.default_rng(5).standard_normal(n)).cuda()
    x = torch.full_like(b, 3.0)
    rep, launches = solve(pkg, device_api, m, torch.zeros_like(b), x)  # solved by x = 0
    assert (rep.iterations, rep.converged, rep.initial_residual, rep.final_residual) == (0, 1, 0.0, 0.0)
    assert launches <= 4 and not torch.any(x)
    rep, _ = solve(pkg, device_api, m, b, x, tolerance=1e-10)
    assert rep.converged == 1 and rep.iterations > 0
    solved = x.clone()
    guess = dict(use_initial_guess=1, convergence=pkg.abi.CONVERGENCE_ABSOLUTE, tolerance=2.0 * rep.final_residual)
    again, launches = solve(pkg, device_api, m, b, x, **guess)  # a guess that is good enough
    assert (again.iterations, again.converged) == (0, 1) and launches <= 4
    assert again.initial_residual == again.final_residual and torch.equal(x, solved)
    for use in (0, 1):  # no iterations allowed
        x.copy_(solved)
        rep, launches = solve(pkg, device_api, m, b, x, max_iters=0, use_initial_guess=use, tolerance=0.0)
        assert (rep.iterations, rep.converged) == (0, 0) and launches <= 4
        assert torch.equal(x, solved if use else torch.zeros_like(x))


def test_little_to_do(pkg, device_api):
    # 120,000 rows: a step is four launches, up to two steps beyond the first may be queued, and a cycle has three more
    import torch

    n = 120000
    keep, m = system(pkg, n)
    b = torch.as_tensor(np.random.default_rng(5).standard_normal(n)).cuda()
    most = []
    for _ in range(3):
        rep, launches = solve(pkg, device_api, m, b, torch.zeros_like(b), tolerance=0.1)
        assert rep.iterations == 1 and rep.converged == 1
        most.append(launches)
    assert min(most) <= 3 * 4 + 4, most


def test_a_matrix_with_nan(pkg, device_api):
    import torch

    keep, m = system(pkg, 3000, bad=True)
    x = torch.zeros(3000, dtype=torch.float64, device="cuda")
    rep, _ = solve(pkg, device_api, m, torch.zeros_like(x), x, max_iters=5)
    assert rep.converged == 0 and np.isnan(rep.final_residual) and bool(torch.isnan(x).all())
