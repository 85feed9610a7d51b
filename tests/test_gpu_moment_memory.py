"""The moment stage's scratch (csrc/context.cu): what lsmps_ctx_reserve sets aside for it in each form."""

import pytest

pytestmark = pytest.mark.gpu


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
