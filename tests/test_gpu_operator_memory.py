"""What the operators' deterministic backward holds on the device (include/lsmps_b200.h): 64 bytes per entry and 72 per
particle of scratch with at most 256 MiB to grow, beside the inverses and records of the pair."""

import pytest

import test_gpu_adjoint as fluid_pair

pytestmark = pytest.mark.gpu


def test_backward_scratch(pkg, device_api):
    import torch

    case = pkg.cases.lattice_box(n=64, l0=0.01)
    ops = fluid_pair.Operators(pkg, device_api, case)
    f, v = fluid_pair.fields(pkg, case)
    x = [torch.from_numpy(case.fluid[k].copy()).cuda() for k in ("x", "y", "z")]
    f, v = torch.from_numpy(f).cuda(), [torch.from_numpy(a.copy()).cuda() for a in v]
    cot = fluid_pair.cotangents(pkg, ops)
    ops.backward(x, f, v, cot)  # the calling code's own tensors
    keep = ops.ctx
    torch.cuda.synchronize()
    keep.close()
    before = torch.cuda.mem_get_info()[0]
    ops.ctx = device_api.Context(0)
    ops.backward(x, f, v, cot)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    ops.ctx.close()
    n, k = ops.n, ops.k
    assert k > 20_000_000  # a quarter of the records is more than the growth allowed
    # inverse, trace, regularisation, info: 668 bytes a particle; two packs 64; moment sums 280; 32 MB of granules
    assert held <= 64 * k + (72 + 668 + 64 + 280) * n + (256 << 20) + (32 << 20), (held, k)
