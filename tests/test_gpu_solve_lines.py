"""The solve on both sides of 2,048 rows, above which the product and its dot products are two kernels (csrc/solve.cu), at
every basis width: as test_gpu_solve_shapes.py's widths."""

import pytest

import test_gpu_solve_shapes as shapes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,restart", [(2048, 20), (2049, 20), (2049, 8), (2049, 25), (2500, 64), (40000, 16)])
def test_widths(pkg, device_api, oracle, n, restart):
    shapes.test_widths(pkg, device_api, oracle, n, restart)
