"""Which launch shapes a grid runs with: the ones it starts with on either side of each line, with the
bits of one tile per CTA throughout, and what the autotuner may pick."""
from __future__ import annotations

import numpy as np
import pytest

from cirrus_b200 import KERNEL_GS_SWEEP, KERNEL_LAPLACIAN, KERNEL_PRESMOOTH, KERNEL_PROLONG_SWEEP, KERNEL_RESIDUAL_RESTRICT, DeviceGrid, GMGSolver, workloads as W

pytestmark = pytest.mark.gpu

VCYCLE = (KERNEL_GS_SWEEP, KERNEL_PRESMOOTH, KERNEL_PROLONG_SWEEP, KERNEL_RESIDUAL_RESTRICT)
WIDE = 6              # 256 threads per tile
PLAIN = 4             # one tile per 128-thread CTA
LARGE, LARGE_LAP = 9, 16  # two (the Laplacian: four) tiles per group, prefetching
SMALL_GRID = 16384    # tiles up to which the wide kernels serve a grid
WIDE_TILES = 1024     # and those of a level up to which they serve it


def shapes(g, kernel, levels):
    return [g.get_launch_shape(kernel, l) for l in range(levels)]


@pytest.mark.parametrize("name,copies", [
    ("sphere256", 2),        # a small grid with wide levels, one of 1025 to 5119 tiles and a large one
    ("sphere256", 3),        # no wide levels
    ("uniform128", 1),       # 512 and 4096 tiles: wide and plain
    ("uniform128", 2),       # levels of 1024 (wide) and 8192 tiles: the sweep's line exactly
    ("uniform64", 16),       # 1024 (wide) and 8192
    ("uniform64", 17),       # 1088 and 8704, either side
])
def test_default_shapes(name, copies, built_cache):
    topo = (W.build(W.uniform(3)) if name == "uniform64" else built_cache(name)).topology
    tiles = topo.tiles()
    g = DeviceGrid([topo] * copies)
    levels = int(tiles[:, 0].max()) + 1
    for l in range(levels):
        n = copies * int(((tiles[:, 0] == l) & (tiles[:, 4] != W.GHOST)).sum())
        small = WIDE if g.num_tiles <= SMALL_GRID and n <= WIDE_TILES else PLAIN
        want = {KERNEL_PROLONG_SWEEP: small, KERNEL_GS_SWEEP: LARGE if n >= 8192 else small,
                KERNEL_PRESMOOTH: LARGE if n >= 5120 else small, KERNEL_RESIDUAL_RESTRICT: LARGE if n >= 5120 else small}
        for k, shape in want.items():
            assert g.get_launch_shape(k, l) == shape, (l, n, k)
    leafs = copies * int(((tiles[:, 4] & W.LEAF) != 0).sum())
    assert g.get_launch_shape(KERNEL_LAPLACIAN) == (LARGE_LAP if leafs >= 8192 else PLAIN)
    rng = np.random.default_rng(1)
    b = rng.standard_normal((len(tiles), 512)).astype(np.float32) * ((topo.cell_types() & W.INTERIOR) != 0) * ((tiles[:, 4] & W.LEAF) != 0)[:, None]
    out = []
    for pin in (False, True):
        if pin:
            g.set_launch_shape(PLAIN)
        for i in range(copies):
            g.set_channel_instance(i, 1, b * np.float32(i + 1))
        GMGSolver().solve_batch(g, max_iters=3)
        out.append([g.get_channel_instance(i, 0).view(np.uint32) for i in range(copies)])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
    g.close()


def test_autotuner_keeps_the_wide_kernels_to_small_grids(built_cache):
    b = built_cache("sphere256")
    levels = int(b.tiles[:, 0].max()) + 1
    g = DeviceGrid([b.topology] * 3)
    assert g.num_tiles > SMALL_GRID
    g.autotune(reps=5)
    for k in VCYCLE:
        assert WIDE not in shapes(g, k, levels), k
    g.close()
