"""Scratch that a context allocates on one stream and first uses on another, with nothing waited for in between
(lsmps_ctx_reserve, then lsmps_ctx_set_stream): the list of particles with walls (csrc/moment.cu) has to start empty in
every call by that call's own work.  The first stream is kept busy meanwhile, so that what reserve might have queued there
would come late."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("inverse_matrices", "moment_trace", "regularization_added", "info")


@pytest.mark.parametrize("nx", [8, 24], ids=["parts", "threads"])
def test_reserve_then_another_stream(pkg, device_api, nx):
    import torch

    case = pkg.cases.CASES["dam_break_shuffled"](nx=nx, ny=8, nz=nx, l0=0.005)
    dev = device_api.device_buffers(case)
    ctx = device_api.Context(0)
    kinds = [0, 1]
    try:
        ctx.build_neighbor_lists(dev, case.params)
        ctx.prepare_moments(dev, case.params, kinds)
    finally:
        ctx.close()
    want = {(k, f): dev.alloc.to_numpy(dev.moments[k][f]).copy() for k in kinds for f in KEYS}
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    a = torch.ones(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        for k in kinds:
            for f in KEYS:
                dev.moments[k][f].zero_()
        torch.cuda.synchronize()
        ctx = device_api.Context(0, synchronous=False, use_torch_stream=False)
        try:
            ctx.set_stream(first.cuda_stream)
            with torch.cuda.stream(first):
                for _ in range(20):
                    a = torch.matmul(a, a).clamp_(-1.0, 1.0)
            ctx.reserve(dev.n_fluid, dev.n_wall, dev.n_cells)
            ctx.set_stream(second.cuda_stream)
            for _ in range(2):
                ctx.prepare_moments(dev, case.params, kinds)
            ctx.synchronize()
            torch.cuda.synchronize()
        finally:
            ctx.close()
        for (k, f), w in want.items():
            assert np.array_equal(dev.alloc.to_numpy(dev.moments[k][f]), w, equal_nan=True), (k, f)
