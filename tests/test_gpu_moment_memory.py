"""The moment stage's scratch (csrc/context.cu): what lsmps_ctx_reserve sets aside for it in each form, and a capture of the
moment stage on a context whose packs other calls have grown but that has no sums yet."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("inverse_matrices", "moment_trace", "regularization_added", "info")


def reserved(pkg, api, precision, n):
    import torch

    ctx = api.Context(0, precision=precision)
    try:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ctx.reserve(n, 1000, 1000)
        return (before - torch.cuda.mem_get_info()[0]) / n
    finally:
        ctx.close()


def test_reserve(pkg, device_api):
    """The mixed form holds its operator rows, 2 x (36 floats + 36 doubles + a byte + an int) a particle, and no wall terms,
    which the plain form has 612 bytes of; the sums and the rest are the same.  (2 MB allocation granules: 20 bytes a
    particle in all.)"""
    n = 1000000
    plain = reserved(pkg, device_api, pkg.abi.PRECISION_PLAIN, n)
    mixed = reserved(pkg, device_api, pkg.abi.PRECISION_MIXED, n)
    assert abs(mixed - plain - (2 * (36 * 4 + 36 * 8 + 1 + 4) - (76 * 8 + 4))) < 20, (plain, mixed)


@pytest.mark.parametrize("earlier", [False, True], ids=["first", "larger"])
def test_capture_without_sums(pkg, device_api, earlier):
    import torch

    case = pkg.cases.CASES["dam_break_shuffled"](nx=20, ny=8, nz=20, l0=0.005)
    dev = device_api.device_buffers(case)
    kinds = [0, 1, 3]
    ctx = device_api.Context(0, synchronous=False)
    stream = torch.cuda.Stream()
    try:
        ctx.build_neighbor_lists(dev, case.params)
        ctx.classify_surface(dev, case.params)  # grows the packs
        if earlier:  # sums and terms of a smaller set first
            small = pkg.cases.lattice_box(n=4, l0=0.01)
            other = device_api.device_buffers(small)
            ctx.build_neighbor_lists(other, small.params)
            ctx.prepare_moments(other, small.params, kinds)
        dev.params_for_moment = case.params
        for k in kinds:
            dev.moment_view(k)
        ctx.synchronize()
        torch.cuda.synchronize()
        ctx.set_stream(stream.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.prepare_moments(dev, case.params, kinds)
        with torch.cuda.stream(stream):
            graph.replay()
            graph.replay()
        torch.cuda.synchronize()
        got = {(k, f): dev.alloc.to_numpy(dev.moments[k][f]).copy() for k in kinds for f in KEYS}
        ctx.prepare_moments(dev, case.params, kinds)
        ctx.synchronize()
        torch.cuda.synchronize()
        for (k, f), g in got.items():
            assert np.array_equal(g, dev.alloc.to_numpy(dev.moments[k][f]), equal_nan=True), (k, f)
        assert np.any(got[0, "moment_trace"] != got[3, "moment_trace"])
        del graph
    finally:
        ctx.close()
