"""Any output pointer of the operator pairs' forward may be NULL (include/lsmps_b200.h): every output asked for alone has
the bits it has when all are asked for, and nothing else is written."""

import numpy as np
import pytest

import test_gpu_adjoint as fluid_pair
import test_gpu_step_adjoint as step_pair

pytestmark = pytest.mark.gpu


def each_alone(ops, forward):
    full = ops.alloc_out

    def only(names):
        ops.alloc_out = lambda: {k: v.fill_(-7) for k, v in full().items() if k in names}
        return {k: v.cpu().numpy() for k, v in forward().items()}

    want = only(set(full()))
    for name, w in want.items():
        assert np.any(w != -7), name
        assert np.array_equal(only({name})[name], w), name
    pair = only({"grad_y", "ppe_rhs"})
    assert np.array_equal(pair["grad_y"], want["grad_y"]) and np.array_equal(pair["ppe_rhs"], want["ppe_rhs"])


def test_fluid_pair(pkg, device_api):
    import torch

    case = pkg.cases.lattice_box(n=6, l0=0.01)
    ops = fluid_pair.Operators(pkg, device_api, case)
    f, v = fluid_pair.fields(pkg, case)
    x = [torch.from_numpy(case.fluid[k].copy()).cuda() for k in ("x", "y", "z")]
    f, v = torch.from_numpy(f).cuda(), [torch.from_numpy(a.copy()).cuda() for a in v]
    each_alone(ops, lambda: ops.forward(x, f, v))


def test_step_pair(pkg, device_api):
    ops = step_pair.StepOps(pkg, device_api, pkg.cases.lattice_box(n=6, l0=0.01))
    each_alone(ops, ops.forward)
