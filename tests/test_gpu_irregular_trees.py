"""Trees that spawning and refining never make but an import accepts: a tile under a GHOST tile, a
NONLEAF tile short of a child, a LEAF tile with LEAF children; and cells of no or of several types.
They take the general forms of the steps around the solve (bit for bit against the CPU oracle) and of
the AMG V-cycle (launch for launch those of the unfused one, where a regular tree takes fewer)."""
from __future__ import annotations

import numpy as np
import pytest

from cirrus_b200 import AMGSolver, DeviceGrid, Topology, workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def kids(l, x, y, z):
    return [(l + 1, 2 * x + (o & 1), 2 * y + (o >> 1 & 1), 2 * z + (o >> 2), W.LEAF) for o in range(8)]


# two coarse tiles, the right one refined; GHOST tiles over the left one's right half
COARSE = [(0, 0, 0, 0, W.LEAF), (0, 1, 0, 0, W.NONLEAF)]
GHOSTS = [(1, 1, y, z, W.GHOST) for y in (0, 1) for z in (0, 1)]
TREES = {
    "regular": COARSE + kids(0, 1, 0, 0) + GHOSTS,
    "tile under a GHOST tile": COARSE + kids(0, 1, 0, 0) + GHOSTS + [(2, 3, 0, 0, W.LEAF), (2, 3, 2, 1, W.LEAF)],
    "NONLEAF tile short of a child": COARSE + kids(0, 1, 0, 0)[1:] + GHOSTS,
    "LEAF tile with LEAF children": COARSE + kids(0, 1, 0, 0) + GHOSTS[1:] + [(1, 1, 0, 0, W.LEAF), (1, 0, 1, 1, W.LEAF)],
}


def build(rows, seed, types=(W.DIRICHLET, W.INTERIOR, W.NEUMANN), p=(0.05, 0.85, 0.1)):
    t = Topology(0.125, W.FLUID_EULER_LOG2_HASH)
    for l, x, y, z, kind in rows:
        t.set_tile(l, (x, y, z), kind)
    t.compress()
    rng = np.random.default_rng(seed)
    t.set_cell_types(rng.choice(np.array(types, dtype=np.uint8), (t.num_tiles, 512), p=p))
    t.calc_cell_types_from_leafs()
    return t, rng


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def check_projection_steps(t, rng):
    tiles = t.tiles()
    leaf = (tiles[:, 4] & W.LEAF) != 0
    f = O.CpuOracle(tiles)
    f.set_ctypes(t.cell_types())
    g = DeviceGrid(t)
    u = rng.standard_normal((3, len(tiles), 512)).astype(np.float32) * leaf[None, :, None]
    for a in range(3):
        g.set_channel(6 + a, u[a])
    g.projection_rhs()
    assert np.array_equal(bits(g.get_channel(1)), bits(f.rhs(u)))
    p = rng.standard_normal((len(tiles), 512)).astype(np.float32) * leaf[:, None]
    u = rng.standard_normal((3, len(tiles), 512)).astype(np.float32)
    g.set_channel(0, p)
    for a in range(3):
        g.set_channel(6 + a, u[a])
    g.add_gradient_to_face_centers()
    _, want = f.add_gradient(p, u)
    for a in range(3):
        assert np.array_equal(bits(g.get_channel(6 + a)), bits(want[a])), a
    g.close()


@pytest.mark.parametrize("seed", [1, 2])
@pytest.mark.parametrize("name", sorted(TREES))
def test_projection_steps(name, seed):
    check_projection_steps(*build(TREES[name], seed))


@pytest.mark.parametrize("types", [(1, 2, 3), (0, 1, 2, 3, 4, 5, 6, 7)])
def test_cells_of_several_types(types):
    p = np.full(len(types), 0.5 / (len(types) - 1))
    p[types.index(W.INTERIOR)] = 0.5
    check_projection_steps(*build(TREES["regular"], 5, types, p))


@pytest.mark.parametrize("name", sorted(TREES))
def test_amg_vcycle(name, monkeypatch):
    t, rng = build(TREES[name], 3)
    leaf = (t.tiles()[:, 4] & W.LEAF) != 0
    b = rng.standard_normal((t.num_tiles, 512)).astype(np.float32) * ((t.cell_types() & W.INTERIOR) != 0) * leaf[:, None]
    out = {}
    for form in ("default", "generic"):
        if form == "generic":
            monkeypatch.setenv("CIRRUS_VCYCLE", form)
        else:
            monkeypatch.delenv("CIRRUS_VCYCLE", raising=False)
        g, s = DeviceGrid(t), AMGSolver()
        s.prepare_types_and_coeffs(g)
        g.set_channel(1, b)
        out[form] = s.solve_batch(g, max_iters=6), bits(g.get_channel(0)), s.last_result.kernel_launches
        g.close()
    (a, x, n), (e, y, m) = out["default"], out["generic"]
    assert a[0][0] == e[0][0] and np.array_equal(x, y)
    assert (n < m) if name == "regular" else (n == m)
