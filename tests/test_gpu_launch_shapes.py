"""Which launch shapes a grid runs with: what the autotuner may pick by the grid's size."""
from __future__ import annotations

import pytest

from cirrus_b200 import KERNEL_GS_SWEEP, KERNEL_PRESMOOTH, KERNEL_PROLONG_SWEEP, KERNEL_RESIDUAL_RESTRICT, DeviceGrid

pytestmark = pytest.mark.gpu

VCYCLE = (KERNEL_GS_SWEEP, KERNEL_PRESMOOTH, KERNEL_PROLONG_SWEEP, KERNEL_RESIDUAL_RESTRICT)
WIDE = 6              # 256 threads per tile
SMALL_GRID = 16384    # tiles up to which the wide kernels serve a grid


def shapes(g, kernel, levels):
    return [g.get_launch_shape(kernel, l) for l in range(levels)]


def test_autotuner_keeps_the_wide_kernels_to_small_grids(built_cache):
    b = built_cache("sphere256")
    levels = int(b.tiles[:, 0].max()) + 1
    g = DeviceGrid([b.topology] * 3)
    assert g.num_tiles > SMALL_GRID
    g.autotune(reps=5)
    for k in VCYCLE:
        assert WIDE not in shapes(g, k, levels), k
    g.close()
