"""Sizes at which the operator pairs' row kernels change course (csrc/operators.cu):

* rows longer than the 128 entries a warp holds at a time, and particle counts that are no multiple of a block's
  four, against torch FP64 autograd of the same operators (the restatements and tolerances of test_gpu_adjoint.py
  and test_gpu_step_adjoint.py);
* the deterministic backward in several passes over the neighbours (the bounds-checked build's passes are 1 MB of
  records): the same bits as in one pass.
"""

import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import test_gpu_adjoint as fluid_pair
import test_gpu_step_adjoint as step_pair

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def lattice(pkg, n, ratio):
    """lattice_box with support radius ratio * l0 (the cell grid follows)."""
    case = pkg.cases.lattice_box(n=n, l0=0.01)
    p, f, w = case.params, case.fluid, case.walls
    p.support_radius = p.grid.cell_size = ratio * case.l0
    pkg.cases.derive_grid(p, [f["x"], w["x"]], [f["y"], w["y"]], [f["z"], w["z"]])
    return case


def close(got, want, rtol, name):
    err = np.max(np.abs(got - want)) / max(np.max(np.abs(want)), 1e-300)
    assert err < rtol, (name, err)


@pytest.mark.parametrize("n,ratio", [(3, 3.1), (5, 3.1), (7, 4.1)], ids=["27", "125", "343-long-rows"])
def test_fluid_pair(pkg, device_api, n, ratio):
    import torch

    case = lattice(pkg, n, ratio)
    ops = fluid_pair.Operators(pkg, device_api, case)
    longest = int(np.max(np.diff(ops.off)))
    assert (longest > 128) == (ratio > 4), longest
    f_np, v_np = fluid_pair.fields(pkg, case)
    x = [torch.from_numpy(case.fluid[k].copy()).cuda() for k in ("x", "y", "z")]
    f, v = torch.from_numpy(f_np).cuda(), [torch.from_numpy(a.copy()).cuda() for a in v_np]
    out = ops.forward(x, f, v)
    cot = fluid_pair.cotangents(pkg, ops)
    fbar, vbar, xbar = ops.backward(x, f, v, cot)
    xr = torch.from_numpy(np.stack([case.fluid[k] for k in ("x", "y", "z")], 1).copy()).requires_grad_(True)
    fr = torch.from_numpy(f_np.copy()).requires_grad_(True)
    vr = [torch.from_numpy(a.copy()).requires_grad_(True) for a in v_np]
    ref = fluid_pair.torch_operators(xr, fr, vr, ops.off, ops.idx, ops.p)
    for k, r in ref.items():
        close(out[k].cpu().numpy(), r.detach().numpy(), fluid_pair.FORWARD_RTOL, k)
    sum((cot[k].cpu() * r).sum() for k, r in ref.items()).backward()
    for c in range(3):
        close(vbar[c].cpu().numpy(), vr[c].grad.numpy(), fluid_pair.ADJOINT_RTOL, f"v{c}")
        close(xbar[c].cpu().numpy(), xr.grad[:, c].numpy(), fluid_pair.ADJOINT_RTOL, f"x{c}")
    close(fbar.cpu().numpy(), fr.grad.numpy(), fluid_pair.ADJOINT_RTOL, "f")


@pytest.mark.parametrize("n,ratio", [(5, 3.1), (7, 4.1)], ids=["125", "343-long-rows"])
def test_step_pair(pkg, device_api, n, ratio):
    import torch

    case = lattice(pkg, n, ratio)
    ops = step_pair.StepOps(pkg, device_api, case)
    assert (int(np.max(np.diff(ops.off))) > 128) == (ratio > 4)
    out = ops.forward()
    cot = ops.cotangents()
    ub, pb, xb = ops.backward(cot)
    u, p, uw = step_pair.fields(case)
    f, w = case.fluid, case.walls
    xr = torch.from_numpy(np.stack([f[k] for k in ("x", "y", "z")], 1).copy()).requires_grad_(True)
    ur = torch.from_numpy(u.copy()).requires_grad_(True)
    pr = torch.from_numpy(p.copy()).requires_grad_(True)
    xw = torch.from_numpy(np.stack([w[k] for k in ("x", "y", "z")], 1).copy())
    nw = torch.from_numpy(np.stack([w[k] for k in ("normal_x", "normal_y", "normal_z")], 1).copy())
    ref = step_pair.torch_step_operators(xr, ur, pr, xw, nw, torch.from_numpy(uw.copy()), ops.off, ops.idx, ops.woff,
                                         ops.widx, ops.labels, ops.p)
    for k, r in ref.items():
        close(out[k].cpu().numpy(), r.detach().numpy(), step_pair.FORWARD_RTOL, k)
    sum((cot[k].cpu() * r).sum() for k, r in ref.items()).backward()
    for c in range(3):
        close(ub[c].cpu().numpy(), ur.grad[:, c].numpy(), step_pair.ADJOINT_RTOL, f"u{c}")
        close(xb[c].cpu().numpy(), xr.grad[:, c].numpy(), step_pair.ADJOINT_RTOL, f"x{c}")
    close(pb.cpu().numpy(), pr.grad.numpy(), step_pair.ADJOINT_RTOL, "p")


CHILD = textwrap.dedent(r"""
    import sys, importlib
    sys.path[:0] = [ROOT, ROOT + "/tests"]
    import numpy as np, torch
    import __graft_entry__ as ge
    pkg = ge.load_package()
    api = importlib.import_module("lsmps3d_b200.api")
    import test_gpu_step_adjoint as step_pair
    ops = step_pair.StepOps(pkg, api, pkg.cases.lattice_box(n=16, l0=0.01))
    ub, pb, xb = ops.backward(ops.cotangents())
    np.savez(OUT, entries=np.array([ops.k]), *[t.cpu().numpy() for t in (*ub, pb, *xb)])
""")


def test_backward_in_passes(pkg, device_api, tmp_path):
    got = []
    for name in (pkg.abi.LIB_NAME, pkg.abi.CHECKED_LIB_NAME):
        out = str(tmp_path / (name + ".npz"))
        lib = os.path.join(pkg.abi.PKG_DIR, name)
        if not os.path.exists(lib):
            import importlib

            importlib.import_module("lsmps3d_b200.build").build_all(bounds_check=True)
        subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\nOUT = {out!r}\n" + CHILD], check=True, timeout=600,
                       env=dict(os.environ, LSMPS_B200_LIBRARY=lib))
        got.append(np.load(out))
    assert int(got[0]["entries"][0]) * 64 > 4 << 20  # at least five passes
    for k in got[0].files:
        assert np.array_equal(got[0][k], got[1][k]), k
