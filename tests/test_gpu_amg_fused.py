"""The fused AMG V-cycle of the solves against the one-kernel-per-step V-cycle: the same iterations
and the same pressure bits over trees of every depth, coarse grids of one to eight tiles per
instance, cell types of all kinds (walls, open cells, cells without any open face beside them), and
other restriction and prolongation coefficients; trees it does not take still solve."""
from __future__ import annotations

import numpy as np
import pytest

from cirrus_b200 import AMGSolver, DeviceGrid, Topology, workloads as W

pytestmark = pytest.mark.gpu


def tree(roots, masks, seed):
    t = Topology(0.125, W.FLUID_EULER_LOG2_HASH)
    for r in roots:
        t.set_tile(0, r, W.LEAF)
    t.compress()
    t.spawn_ghost_tiles()
    t.iterative_refine(masks=masks)
    tiles, nbr = t.tiles(), t.neighbor_tiles()
    w = W.Workload("test", list(roots), (1, 1, 1), masks, log2_hash=W.FLUID_EULER_LOG2_HASH)
    ct = W.leaf_cell_types(w, tiles, nbr)
    rng = np.random.default_rng(seed)
    leaf = (tiles[:, 4] & W.LEAF) != 0
    solid = (rng.random(ct.shape) < 0.05) & leaf[:, None] & (ct == W.INTERIOR)
    ct[solid] = rng.choice(np.array([W.NEUMANN, W.DIRICHLET], dtype=np.uint8), int(solid.sum()), p=(0.8, 0.2))
    t.set_cell_types(ct)
    t.calc_cell_types_from_leafs()
    b = rng.standard_normal((len(tiles), 512)).astype(np.float32) * ((t.cell_types() & W.INTERIOR) != 0) * leaf[:, None]
    return t, b


def roots_of(n):
    return [(i % 2, (i // 2) % 2, i // 4) for i in range(n)]


def corner_masks(roots, levels, seed):
    """Random refinement, denser towards the origin, level by level."""
    rng = np.random.default_rng(seed)
    ext = np.max(np.array(roots), axis=0) + 1
    return [(rng.random(tuple(ext << l)) < 0.4).astype(np.uint8) for l in range(levels)] + [None] * (10 - levels)


def solve(grid, bs, monkeypatch, generic, **kw):
    if generic:
        monkeypatch.setenv("CIRRUS_VCYCLE", "generic")
    else:
        monkeypatch.delenv("CIRRUS_VCYCLE", raising=False)
    s = AMGSolver(one_over_alpha=kw.pop("one_over_alpha", 1.0), prolong_coeff=kw.pop("prolong_coeff", 1.0))
    s.prepare_types_and_coeffs(grid)
    for i, b in enumerate(bs):
        grid.set_channel_instance(i, 1, b)
        grid.set_channel_instance(i, 0, np.zeros_like(b))
    res = s.solve_batch(grid, max_iters=12, **kw)
    return res, [grid.get_channel_instance(i, 0).view(np.uint32) for i in range(len(bs))], s.last_result.kernel_launches


@pytest.mark.parametrize("nroots,levels,seed", [(1, 1, 1), (1, 3, 2), (2, 2, 3), (5, 2, 4), (8, 1, 5), (9, 1, 6)])
def test_fused_equals_generic(nroots, levels, seed, monkeypatch):
    roots = roots_of(nroots)
    t, b = tree(roots, corner_masks(roots, levels, seed), seed)
    g = DeviceGrid([t])
    a = solve(g, [b], monkeypatch, False)
    e = solve(g, [b], monkeypatch, True)
    assert a[0] == e[0] and np.array_equal(a[1][0], e[1][0])
    assert (a[2] < e[2]) == (nroots <= 8)  # nine coarse tiles: the generic V-cycle either way
    g.close()


@pytest.mark.parametrize("kw", [{"one_over_alpha": 0.5}, {"prolong_coeff": 1.5}, {"coarsest_iters": 3}, {"coarsest_iters": 2},
                                {"pure_neumann": [True, False, True]}, {"active": [True, False, True]}, {"level_iters": 2}])
def test_fused_batch_options(kw, monkeypatch):
    built = [tree(roots_of(n), corner_masks(roots_of(n), lv, n), n) for n, lv in ((1, 3), (3, 1), (2, 2))]
    g = DeviceGrid([t for t, _ in built])
    bs = [b for _, b in built]
    a = solve(g, bs, monkeypatch, False, **dict(kw))
    e = solve(g, bs, monkeypatch, True, **dict(kw))
    assert a[0] == e[0]
    for x, y in zip(a[1], e[1]):
        assert np.array_equal(x, y)
    g.close()
