"""The steps on either side of the solve, bit for bit against the CPU oracle, on trees of cells of
every type (solid, open and fluid at random, so that every face rule is met at tile, level and
domain boundaries): face clearing and propagation with the divergence, alone and as the one call,
and the velocity update; and the update where h is no power of two, against the same operations in
NumPy's single precision."""
from __future__ import annotations

import numpy as np
import pytest

from cirrus_b200 import DeviceGrid, Topology, workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def random_types(b, seed, share):
    """The workload's topology with a share of its LEAF cells turned solid or open."""
    rng = np.random.default_rng(seed)
    ct = b.ctypes.copy()
    leaf = (b.tiles[:, 4] & W.LEAF) != 0
    turn = (rng.random(ct.shape) < share) & leaf[:, None]
    ct[turn] = rng.choice(np.array([W.NEUMANN, W.DIRICHLET], dtype=np.uint8), int(turn.sum()))
    t = W.build(b.workload).topology
    t.set_cell_types(ct)
    t.calc_cell_types_from_leafs()
    return t, t.cell_types(), rng


@pytest.mark.parametrize("share", [0.0, 0.02, 0.5])
@pytest.mark.parametrize("name", ["uniform32_small", "sphere64_small", "ring64_small"])
def test_projection_steps_bitwise(name, share, built_cache):
    b = built_cache(name)
    topo, ct, rng = random_types(b, 3, share)
    leaf = (b.tiles[:, 4] & W.LEAF) != 0
    u = rng.standard_normal((3, len(b.tiles), 512)).astype(np.float32) * leaf[None, :, None]
    f = O.CpuOracle(b.tiles)
    f.set_ctypes(ct)
    want = f.rhs(u)
    grids = [DeviceGrid(topo), DeviceGrid(topo)]
    for g in grids:
        for a in range(3):
            g.set_channel(6 + a, u[a])
    grids[0].projection_rhs()
    grids[1].clear_neumann_neighbor_faces()
    for a in range(3):
        grids[1].propagate_to_children(6 + a)
    grids[1].velocity_volume_divergence_on_leafs()
    for c in (1, 6, 7, 8):
        assert np.array_equal(bits(grids[0].get_channel(c)), bits(grids[1].get_channel(c))), c
    assert np.array_equal(bits(grids[0].get_channel(1)), bits(want))
    p = rng.standard_normal((len(b.tiles), 512)).astype(np.float32) * leaf[:, None]
    u = rng.standard_normal((3, len(b.tiles), 512)).astype(np.float32)
    g = grids[0]
    g.set_channel(0, p)
    for a in range(3):
        g.set_channel(6 + a, u[a])
    g.add_gradient_to_face_centers()
    op, ou = f.add_gradient(p, u)
    ghost = (b.tiles[:, 4] & W.GHOST) != 0
    assert np.array_equal(bits(g.get_channel(0))[ghost], bits(op)[ghost])
    for a in range(3):
        assert np.array_equal(bits(g.get_channel(6 + a)), bits(ou[a])), a


@pytest.mark.parametrize("h0", [0.1, 0.125, 3.0])
def test_gradient_voxel_sizes(h0):
    t = Topology(h0, W.FLUID_EULER_LOG2_HASH)
    t.set_tile(0, (0, 0, 0), W.LEAF)
    t.compress()
    t.set_cell_types(np.full((1, 512), W.INTERIOR, dtype=np.uint8))
    t.calc_cell_types_from_leafs()
    g = DeviceGrid(t)
    rng = np.random.default_rng(1)
    p = rng.standard_normal((8, 8, 8)).astype(np.float32)
    u = rng.standard_normal((3, 8, 8, 8)).astype(np.float32)
    g.set_channel(0, p)
    for a in range(3):
        g.set_channel(6 + a, u[a])
    g.add_gradient_to_face_centers()
    for a in range(3):
        lower = np.zeros_like(p)  # 0 beyond the domain
        at, at0 = [slice(None)] * 3, [slice(None)] * 3
        at[a], at0[a] = slice(1, None), slice(0, -1)
        lower[tuple(at)] = p[tuple(at0)]
        want = u[a] + (p - lower) / np.float32(h0)
        assert np.array_equal(bits(g.get_channel(6 + a)).reshape(8, 8, 8), bits(want)), a
