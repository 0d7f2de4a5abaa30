"""The work a program has this framework do, as cases that can be timed and compared.

A case is one call (or the few calls of one projection step) of the pressure path on an adaptive
octree grid of 8^3-cell tiles, at the sizes of the benchmark configurations, the tests and the
serving sessions:

  solve     GMG- or AMG-preconditioned CG of one instance, of a batch of instances in one tile pool,
            or of several pools at once; plain FP32 to a recursive residual, or mixed precision to
            an FP64 true residual.  The right-hand side is written to the grid, as a simulator does
            each step, then solved; the pressure comes back.
  project   a whole pressure projection: right-hand side from the face velocities, solve, velocity
            update; the divergence-free velocity comes back.
  rhs       its first part alone: face clearing, propagation to GHOST tiles, divergence.
  gradient  its last part alone: the velocity update from a pressure.
  build     the octree built on the GPU for one refinement target and adapted to another (coarsen,
            refine, GHOST tiles), with its cell types.

Geometries: a uniform grid; leaves refined around a sphere; around a vortex ring in a 1x1x2 domain;
around several random spheres (uneven batches).  Velocities are N(0,1) on LEAF faces.
"""
from __future__ import annotations

import time

import numpy as np
import torch

from cirrus_b200 import AMGSolver, DeviceGrid, DeviceTopology, GMGSolver, PRECISION_FP32, PRECISION_MIXED_FP64, Topology
from cirrus_b200 import workloads as W

LEAF, NONLEAF, GHOST = 1, 2, 4
DIRICHLET, INTERIOR, NEUMANN = 1, 2, 4
MOST_TILES = 170048  # the largest listed case's (32 vortex-ring instances)
TYPICAL_ITERS = 30   # PCG iterations to 1e-6 on these geometries (28-31)


def _case(kind, geometry, base, fine, count=1, pools=1, method="gmg", precision="fp32", tol=1e-6, neumann=False, first=0):
    return {"kind": kind, "geometry": geometry, "base": base, "fine": fine, "count": count, "pools": pools, "method": method,
            "precision": precision, "tol": tol, "neumann": neumann, "first": first}


def listed():
    return [
        # one pressure solve of a small scene (effective 64^3): latency and launches
        dict(_case("solve", "sphere", 1, 3), name="solve_sphere64"),
        # one solve on a uniform 128^3 grid
        dict(_case("solve", "uniform", 4, 4), name="solve_uniform128"),
        # one solve per frame of the vortex-ring scene (effective 512x512x1024)
        dict(_case("solve", "ring", 2, 6), name="solve_ring512"),
        # a frame's projection in a closed box (effective 256^3, pure Neumann)
        dict(_case("project", "sphere", 3, 5, neumann=True), name="project_sphere256_neumann"),
        # a batch of simulations advanced together
        dict(_case("solve", "ring", 2, 6, count=8), name="batch_ring512_x8"),
        # the throughput step: 32 instances as four pools solved at once
        dict(_case("solve", "ring", 2, 6, count=8, pools=4), name="pools_ring512_4x8"),
        # FP64-accurate pressure by defect correction
        dict(_case("solve", "ring", 2, 6, count=4, precision="mixed", tol=1e-8), name="mixed_ring512_x4"),
        # an uneven batch, as the serving loop merges sessions of different sizes
        dict(_case("solve", "spheres", 0, 0, count=12, precision="mixed"), name="mixed_spheres_x12"),
        # the AMG preconditioner on a small batch
        dict(_case("solve", "ring", 2, 6, count=4, method="amg"), name="amg_ring512_x4"),
        # right-hand sides and velocity updates of a batch, the steps on either side of its solve
        dict(_case("rhs", "ring", 2, 6, count=8), name="rhs_ring512_x8"),
        dict(_case("gradient", "ring", 2, 6, count=8), name="gradient_ring512_x8"),
        # the grid of a frame built and adapted on the GPU
        dict(_case("build", "ring", 2, 6), name="build_ring512"),
    ]


def draw(rng):
    while True:
        kind = rng.choice(("solve",) * 5 + ("project", "project", "rhs", "gradient", "build"))
        geometry = rng.choice(("uniform", "sphere", "ring", "spheres") if kind in ("solve", "rhs") else ("uniform", "sphere", "ring"))
        base, fine, first = 0, 0, 0
        if geometry == "uniform":
            base = fine = rng.randint(2, 4)
        elif geometry == "sphere":
            fine = rng.randint(3, 5)
            base = rng.randint(max(1, fine - 3), fine - 1)
        elif geometry == "ring":
            fine = rng.randint(3, 6)
            base = rng.randint(1, min(3, fine - 1))
        else:
            first = rng.randint(0, 40)
        count = 1 if kind == "build" else int(round(2 ** rng.uniform(0, 5)))
        method = "amg" if kind == "solve" and rng.random() < 0.2 else "gmg"
        precision = "mixed" if kind == "solve" and method == "gmg" and rng.random() < 0.35 else "fp32"
        tol = rng.choice((1e-6, 1e-8)) if precision == "mixed" else 1e-6
        neumann = kind == "project" and geometry == "sphere" and rng.random() < 0.5  # a closed box
        pools = 1
        if kind == "solve" and count >= 4 and rng.random() < 0.3:
            pools, count = 2, count // 2
        if kind == "project":  # one simulation's step
            count = 1
        if geometry == "spheres":
            count = min(count, 12)
        c = _case(kind, geometry, base, fine, count, pools, method, precision, tol, neumann, first)
        cost = sum(t[0].shape[0] for t in _tiles_of(c)) * pools * (4 if method == "amg" else 2 if precision == "mixed" else 1)
        if cost <= MOST_TILES:
            return c


# ----------------------------------------------------------------------------- grids
def _workload(case, instance):
    g = case["geometry"]
    if g == "uniform":
        return W.uniform(case["fine"])
    if g == "sphere":
        return W.sphere(case["base"], case["fine"], pure_neumann=case["neumann"])
    if g == "ring":
        return W.ring(case["base"], case["fine"])
    return W.random_spheres(case["first"] + instance)


def _topology(w):
    t = Topology(w.h0, w.log2_hash)
    for r in w.roots:
        t.set_tile(0, r, LEAF)
    t.compress()
    t.spawn_ghost_tiles()
    t.iterative_refine(masks=w.masks)
    tiles = t.tiles()
    t.set_cell_types(W.leaf_cell_types(w, tiles, t.neighbor_tiles()))
    t.calc_cell_types_from_leafs()
    return t, tiles, t.cell_types()


def _tiles_of(case):
    """(tiles, cell types) of each instance of one pool; equal instances are built once."""
    same = case["geometry"] != "spheres"
    one = _topology(_workload(case, 0))[1:] if same else None
    return [one if same else _topology(_workload(case, i))[1:] for i in range(case["count"])]


def _topologies(case):
    if case["geometry"] != "spheres":
        return [_topology(_workload(case, 0))] * case["count"]
    return [_topology(_workload(case, i)) for i in range(case["count"])]


class _View:
    """Channels of a grid for torch; the tensor made from it keeps it, and it keeps the grid, alive."""

    def __init__(self, grid, first, shape):
        self.grid = grid
        self.__cuda_array_interface__ = {"data": (grid.channel_ptr(first), False), "shape": shape, "typestr": "<f4", "version": 3}


def _channels(grid, first, count):
    """Channels first..first+count-1 of a grid as a (count, n, 512) tensor on its memory."""
    return torch.as_tensor(_View(grid, first, (count, grid.num_tiles, 512)), device="cuda")


class _Pool:
    """The tables of one pool in the pool's order (level by level, inside a level instance by
    instance), for inputs and for the 64-bit answers."""

    def __init__(self, instances):
        t = np.concatenate([np.concatenate([x[0], np.full((len(x[0]), 1), i, np.int32)], axis=1) for i, x in enumerate(instances)])
        ct = np.concatenate([x[1] for x in instances])
        order = np.argsort(t[:, 0], kind="stable")
        t, ct = t[order].astype(np.int64), ct[order]
        self.n = len(t)
        key = self._key(t[:, 5], t[:, 0], t[:, 1], t[:, 2], t[:, 3])
        by = np.argsort(key)
        find = lambda l, x, y, z: self._find(key, by, self._key(t[:, 5], l, x, y, z), (x < 0) | (y < 0) | (z < 0) | (l < 0))  # noqa: E731
        l, x, y, z = t[:, 0], t[:, 1], t[:, 2], t[:, 3]
        d = ((-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1))
        dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
        self.nb = dev(np.stack([find(l, x + a, y + b, z + c) for a, b, c in d], axis=1))
        self.parent = dev(find(l - 1, x >> 1, y >> 1, z >> 1))
        self.child = dev(np.stack([find(l + 1, 2 * x + (o & 1), 2 * y + (o >> 1 & 1), 2 * z + (o >> 2)) for o in range(8)], axis=1))
        self.octant = dev((x & 1) | (y & 1) << 1 | (z & 1) << 2)
        self.inst, self.level, self.type, self.ct = dev(t[:, 5].copy()), dev(l.copy()), dev(t[:, 4].copy()), dev(ct.astype(np.int64))
        self.h = (0.125 / 2.0 ** self.level.double())[:, None]
        o = torch.arange(512, device="cuda")
        self.ijk = (o >> 6, o >> 3 & 7, o & 7)

    @staticmethod
    def _key(i, l, x, y, z):
        return (((i * 16 + l) * 1024 + x) * 1024 + y) * 1024 + z

    @staticmethod
    def _find(key, by, want, outside):
        at = np.minimum(np.searchsorted(key, want, sorter=by), len(key) - 1)
        got = by[at]
        return np.where((key[got] == want) & ~outside, got, -1)

    def neighbour(self, f):
        """(n, 512): the cell across face f at the same level as a flat index, -1 where its tile is absent;
        and the tile that holds it (own tile inside)."""
        c = list(self.ijk)
        c[f >> 1] = c[f >> 1] + (1 if f & 1 else -1)
        inside = (c[f >> 1] >= 0) & (c[f >> 1] < 8)
        off = (c[0] & 7) * 64 + (c[1] & 7) * 8 + (c[2] & 7)
        tile = torch.where(inside[None], torch.arange(self.n, device="cuda")[:, None], self.nb[:, f:f + 1])
        return torch.where(tile >= 0, tile * 512 + off, -1), tile

    def parents(self):
        """(n, 512): the parent tile's cell over each cell, -1 without a parent tile."""
        b = [((self.octant >> a & 1)[:, None] * 8 + self.ijk[a][None]) >> 1 for a in range(3)]
        return torch.where(self.parent[:, None] >= 0, self.parent[:, None] * 512 + b[0] * 64 + b[1] * 8 + b[2], -1)

    def child_sums(self, v, types):
        """(n, 512): per cell the sum of v over its 2x2x2 children of these types, 0 without a child tile."""
        i, j, k = self.ijk
        tile = self.child[:, (i >> 2) | (j >> 2) << 1 | (k >> 2) << 2]
        tot = torch.zeros_like(v)
        for q in range(8):
            cell = (2 * i + (q & 1) & 7) * 64 + (2 * j + (q >> 1 & 1) & 7) * 8 + (2 * k + (q >> 2) & 7)
            at = (tile.clamp(min=0) * 512 + cell).view(-1)
            ok = (tile >= 0) & ((self.ct.view(-1)[at] & types) != 0).view(tile.shape)
            tot += torch.where(ok, v.reshape(-1)[at].view(tile.shape), 0)
        return tot

    def rows(self, types):
        return ((self.type & types) != 0)[:, None]


def _take(v, at, other=0):
    return torch.where(at >= 0, v.reshape(-1)[at.clamp(min=0)], other)


def _velocity(pool, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    u = torch.randn((3, pool.n, 512), generator=g, device="cuda", dtype=torch.float32)
    return u * pool.rows(LEAF)[None]


def _rhs64(pool, u32):
    """(b, cleared and propagated velocity) of a projection in FP64."""
    u, ct, tt = u32.double(), pool.ct, pool.type[:, None]
    for a in range(3):
        at, tile = pool.neighbour(2 * a)
        ntt = torch.where(tile >= 0, _take(pool.type, tile), 0)
        test = lambda t1: ((ct | t1) & NEUMANN != 0) | (ct & t1 & DIRICHLET != 0)  # noqa: E731
        hit = (ntt & LEAF != 0) & test(_take(ct, at)) | (tile == torch.arange(pool.n, device="cuda")[:, None]) & test(_take(ct, at))
        for q in range(4):  # the finer cells behind a face to a refined neighbour
            c = [2 * pool.ijk[d] for d in range(3)]
            c[a] = torch.full_like(c[a], 15)
            c[(a + 1) % 3] = c[(a + 1) % 3] + (q >> 1)
            c[(a + 2) % 3] = c[(a + 2) % 3] + (q & 1)
            octant = (c[0] >> 3) | (c[1] >> 3) << 1 | (c[2] >> 3) << 2
            fine = pool.child[tile.clamp(min=0), octant[None].expand_as(tile)]
            cell = (c[0] & 7) * 64 + (c[1] & 7) * 8 + (c[2] & 7)
            ok = (tile >= 0) & (ntt & LEAF == 0) & (tile != torch.arange(pool.n, device="cuda")[:, None]) & (fine >= 0)
            hit = hit | ok & test(_take(ct, torch.where(ok, fine * 512 + cell, -1)))
        u[a] = torch.where(hit & pool.rows(LEAF), 0.0, u[a])
    up = pool.parents()
    for a in range(3):
        v = torch.where(_take(ct, up) & 7 != 0, _take(u[a], up), 0.0)
        u[a] = torch.where(pool.rows(GHOST) & (ct & 7 != 0), v, u[a])
    b = torch.zeros_like(u[0])
    for a in range(3):
        for f in (2 * a, 2 * a + 1):
            at, tile = pool.neighbour(f)
            ntt = torch.where(tile >= 0, _take(pool.type, tile), tt)
            ok = (tt == LEAF) & (ntt & (LEAF | GHOST) != 0) | (tt == GHOST) & (ntt == LEAF)
            b += torch.where(ok, -u[a] if f == 2 * a else _take(u[a], at, 0.0), 0.0)
    b = torch.where((ct & INTERIOR != 0) & pool.rows(LEAF | GHOST), b * pool.h ** 2, 0.0)
    more = torch.where((ct & INTERIOR != 0) & pool.rows(LEAF), pool.child_sums(b, INTERIOR), 0.0)
    return b + more, u


def _gradient64(pool, p32, u32):
    """The velocity after the update from pressure p, in FP64."""
    p, u, ct, tt = p32.double(), u32.double(), pool.ct, pool.type[:, None]
    up = pool.parents()
    both = (ct & INTERIOR != 0) & (_take(ct, up) & INTERIOR != 0)
    p = torch.where(pool.rows(GHOST), torch.where(both, _take(p, up), 0.0), p)
    p = torch.where(ct & INTERIOR != 0, p, 0.0)
    for a in range(3):
        at, tile = pool.neighbour(2 * a)
        ntt = torch.where(tile >= 0, _take(pool.type, tile), tt)
        nct = torch.where(tile >= 0, _take(ct, at), ct)
        same = (tt & LEAF != 0) & (ntt & LEAF != 0)
        cross = (tt & LEAF != 0) & (ntt & GHOST != 0) | (tt & GHOST != 0) & (ntt & LEAF != 0)
        term = (same | cross) & ((ct | nct) & NEUMANN == 0)
        v = torch.where(pool.rows(GHOST), 0.0, u[a])
        v = v + torch.where(term, (p - _take(p, at, 0.0)) / (pool.h * torch.where(same, 1.0, 1.5)), 0.0)
        u[a] = torch.where(pool.rows(LEAF | GHOST), v, u[a])
        take = pool.rows(LEAF) & (ct & (INTERIOR | DIRICHLET) != 0)
        u[a] += torch.where(take, 0.25 * pool.child_sums(u[a], INTERIOR | DIRICHLET), 0.0)
    return u


def _solve64(pool, b, neumann, seconds=14.0):
    """The pressure of right-hand side b (FP64), by conjugate gradients on the assembled matrix of
    the LEAF cells; None when that takes too long."""
    began = time.perf_counter()
    ct = pool.ct
    unknown = pool.rows(LEAF) & (ct & INTERIOR != 0)
    m = int(unknown.sum())
    ids = torch.full((pool.n, 512), -1, dtype=torch.int64, device="cuda")
    ids[unknown] = torch.arange(m, device="cuda")
    ids, up = ids.view(-1), pool.parents()
    own = ids.view(pool.n, 512)
    diag = torch.zeros(m, dtype=torch.float64, device="cuda")
    rows, cols, vals = [], [], []

    def couple(on, r, c, w):
        """Row cells r take w * (x_r - x_c); a column that is no unknown holds 0."""
        on = on & (r >= 0)
        r, c, w = r[on], c[on], w[on]
        diag.index_add_(0, r, w)
        on = c >= 0
        rows.append(r[on]), cols.append(c[on]), vals.append(-w[on])

    for f in range(6):
        at, tile = pool.neighbour(f)
        ntt = torch.where(tile >= 0, _take(pool.type, tile), LEAF)
        nct = torch.where(tile >= 0, _take(ct, at), DIRICHLET)
        open_ = pool.rows(LEAF) & ((ct | nct) & NEUMANN == 0)
        w = pool.h.expand(pool.n, 512)
        couple(open_ & (ntt == LEAF), own, _take(ids, at, -1), w)
        coarse = _take(up, at, -1)  # across a GHOST tile: the coarser cell it stands for
        cid = torch.where(nct & INTERIOR != 0, _take(ids, coarse, -1), -1)
        ghost = open_ & (ntt == GHOST)
        couple(ghost, own, cid, w * (2.0 / 3.0))
        couple(ghost, cid, own, w * (2.0 / 3.0))
    i = torch.arange(m, device="cuda")
    a = torch.sparse_coo_tensor(torch.stack([torch.cat(rows + [i]), torch.cat(cols + [i])]), torch.cat(vals + [diag]), (m, m))
    a = a.coalesce().to_sparse_csr()
    r = b.reshape(-1)[unknown.view(-1)].clone()
    if neumann:
        r -= r.mean()
    inv = 1.0 / diag.clamp(min=1e-300)
    x, z = torch.zeros_like(r), r * inv
    p, rz, stop = z.clone(), torch.dot(r, z), 1e-24 * torch.dot(r, r)
    for k in range(60000):
        q = a @ p
        alpha = rz / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        z = r * inv
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
        if k % 50 == 49:
            if bool(torch.dot(r, r) < stop):
                out = torch.zeros(pool.n * 512, dtype=torch.float64, device="cuda")
                out[unknown.view(-1)] = x
                return out.view(pool.n, 512)
            if time.perf_counter() - began > seconds:
                return None
    return None


def _masks(case, seed, moved):
    """Refinement masks of the build case: the feature, or the same a little further on.  The seed
    mirrors the scene in x and y and swaps the two, so that every seed has tiles of its own and as
    many of them."""
    c = np.array((0.53, 0.46, 0.5)) + (0.03 if moved else 0.0)
    if case["geometry"] == "uniform":
        n = 1 << case["fine"] - 1
        masks = [np.ones((1 << l,) * 3, dtype=np.uint8) for l in range(case["fine"])]
        masks[-1][n - n // 4 if moved else n - n // 2:, n - 1:] = 0
        masks += [None] * (10 - case["fine"])
    elif case["geometry"] == "ring":
        masks = W.ring_masks(case["base"], case["fine"], (c[0], c[1], c[2] - 0.25), 0.15, 0.02, 0.1)
    else:
        masks = W.sphere_band_masks(case["base"], case["fine"], c, 0.2, 8 / float(8 << case["fine"]))
    out = []
    for m in masks:
        if m is not None:
            m = m[::-1] if seed & 1 else m
            m = m[:, ::-1] if seed & 2 else m
            m = np.ascontiguousarray(m.transpose(1, 0, 2) if seed & 4 else m)
        out.append(m)
    return out


def _coarsen(masks):
    """CoarsenStep's masks for a refinement target: the tiles whose parent the target leaves unrefined."""
    out = [None] * len(masks)
    for l in range(1, len(masks)):
        if masks[l - 1] is not None:
            out[l] = np.ascontiguousarray(1 - masks[l - 1].repeat(2, 0).repeat(2, 1).repeat(2, 2))
    return out


# ----------------------------------------------------------------------------- the interface
def prepare(case, seed):
    if case["kind"] == "build":
        roots = [(0, 0, 0), (0, 0, 1)] if case["geometry"] == "ring" else [(0, 0, 0)]
        target = _masks(case, seed, True)
        # cell types of the LEAF tiles, mostly fluid, as a scene's solids and open cells would set them
        types = np.random.default_rng(int(seed)).choice(np.array([DIRICHLET, INTERIOR, NEUMANN], dtype=np.uint8), (1024, 512), p=(0.01, 0.95, 0.04))
        return {"case": case, "roots": np.array(roots, dtype=np.int32), "masks": _masks(case, seed, False), "target": target,
                "coarsen": _coarsen(target), "types": np.resize(types, (_built_tiles(case), 512))}
    state = {"case": case, "pools": []}
    for k in range(case["pools"]):
        built = _topologies(case)
        topos = [x[0] for x in built]
        grid = DeviceGrid(topos if len(topos) > 1 else topos[0])
        pool = _Pool([x[1:] for x in built])
        u = _velocity(pool, int(seed) * 1009 + k)
        one = {"grid": grid, "x": _channels(grid, 0, 1)[0], "b": _channels(grid, 1, 1)[0], "u": _channels(grid, 6, 3)}
        if case["kind"] == "solve":
            one["rhs"] = (_rhs64(pool, u)[0] * pool.rows(LEAF)).float()
        else:
            one["velocity"] = u
            one["u"].copy_(u)
        if case["kind"] == "gradient":
            g = torch.Generator(device="cuda").manual_seed(int(seed) + 77)
            one["x"].copy_(torch.randn((pool.n, 512), generator=g, device="cuda") * ((pool.ct & INTERIOR != 0) & pool.rows(LEAF)) * 0.01)
        state["pools"].append(one)
    solver = AMGSolver if case["method"] == "amg" else GMGSolver
    state["solver"] = solver(precision=PRECISION_MIXED_FP64 if case["precision"] == "mixed" else PRECISION_FP32)
    if case["method"] == "amg":
        for one in state["pools"]:
            state["solver"].prepare_types_and_coeffs(one["grid"])
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "build":
        t = DeviceTopology()
        t.set_tiles(0, state["roots"], LEAF)
        t.compress()
        t.spawn_ghost_tiles()
        t.iterative_refine(state["masks"])
        first = t.tiles()
        t.coarsen_step(state["coarsen"])
        t.spawn_ghost_tiles()
        t.iterative_refine(state["target"])
        tiles = t.tiles()
        t.set_cell_types(state["types"] if len(state["types"]) == len(tiles) else np.resize(state["types"], (len(tiles), 512)))
        t.calc_cell_types_from_leafs()
        return {"first": first, "tiles": tiles, "slots": t.hash_slots(), "cell_types": t.cell_types()}
    solver, pools = state["solver"], state["pools"]
    if case["kind"] == "solve":
        for one in pools:
            one["b"].copy_(one["rhs"])
        if len(pools) > 1:
            solver.solve_grids([one["grid"] for one in pools], relative_tolerance=case["tol"])
        elif case["count"] > 1:
            solver.solve_batch(pools[0]["grid"], relative_tolerance=case["tol"])
        else:
            solver.solve(pools[0]["grid"], relative_tolerance=case["tol"]) if case["precision"] == "fp32" else \
                solver.solve_batch(pools[0]["grid"], relative_tolerance=case["tol"])
        return [one["x"] for one in pools]
    one = pools[0]
    if case["kind"] == "rhs":
        one["grid"].projection_rhs()
        return {"b": one["b"], "u": one["u"]}
    one["u"].copy_(one["velocity"])
    if case["kind"] == "project":
        one["grid"].projection_rhs()
        solver.solve(one["grid"], relative_tolerance=case["tol"], is_pure_neumann=case["neumann"])
    one["grid"].add_gradient_to_face_centers()
    return one["u"]


def work(case):
    if case["kind"] == "build":
        # both grids' tile records, then the cell types set, completed and read back
        return {"bytes": _built_tiles(case) * (2 * 20 + 4 + 4 * 512), "flops": 0}
    leaf = mg = ghost = n = 0
    for tiles, _ in _tiles_of(case):
        n += len(tiles)
        leaf += int((tiles[:, 4] == LEAF).sum())
        ghost += int((tiles[:, 4] == GHOST).sum())
        mg += int((tiles[:, 4] != GHOST).sum())
    leaf, mg, ghost, n = (512 * v * case["pools"] for v in (leaf, mg, ghost, n))
    rhs = {"bytes": 13 * (leaf + ghost) + 4 * leaf + 12 * (leaf + ghost), "flops": 12 * (leaf + ghost)}
    grad = {"bytes": 5 * (leaf + ghost) + 24 * leaf + 12 * ghost, "flops": 12 * (leaf + ghost)}
    # per iteration: x, r, p read and written, z written and read, the cell masks; the V-cycle's
    # right-hand sides and corrections of every level
    iters = TYPICAL_ITERS * (1.4 if case["tol"] < 1e-7 else 1.0)
    solve = {"bytes": iters * (33 * leaf + 17 * mg), "flops": iters * (30 * leaf + 60 * mg)}
    if case["kind"] == "solve":
        return solve
    if case["kind"] == "rhs":
        return rhs
    if case["kind"] == "gradient":
        return grad
    return {k: rhs[k] + solve[k] + grad[k] for k in rhs}


def _built_tiles(case):
    """About the tiles of the build case's adapted grid, from the host builder."""
    roots = [(0, 0, 0), (0, 0, 1)] if case["geometry"] == "ring" else [(0, 0, 0)]
    t = Topology()
    for r in roots:
        t.set_tile(0, r, LEAF)
    t.compress()
    t.spawn_ghost_tiles()
    t.iterative_refine(masks=_masks(case, 0, True))
    return t.num_tiles


def tolerance(case):
    if case["kind"] == "build":
        return "exact"
    if case["kind"] in ("rhs", "gradient"):
        return {"rel": 2e-7}
    if case["kind"] == "project":
        return {"rel": 5e-6}
    # an iterative answer: another order of the sums may stop an iteration earlier or later; the
    # answers at these tolerances are up to 2.7e-4 (2.6e-6) from the FP64 ones
    return {"rel": 1e-5 if case["tol"] < 1e-7 else 1e-3}


def exact(case, seed):
    if case["kind"] == "build":
        return None
    out = []
    for k in range(case["pools"]):
        pool = _Pool(_tiles_of(case))
        u = _velocity(pool, int(seed) * 1009 + k)
        if case["kind"] == "rhs":
            b, v = _rhs64(pool, u)
            return {"b": b, "u": v}
        if case["kind"] == "gradient":
            g = torch.Generator(device="cuda").manual_seed(int(seed) + 77)
            p = torch.randn((pool.n, 512), generator=g, device="cuda") * ((pool.ct & INTERIOR != 0) & pool.rows(LEAF)) * 0.01
            return _gradient64(pool, p, u)
        b, v = _rhs64(pool, u)
        if case["kind"] == "solve":
            b = (b * pool.rows(LEAF)).float().double()
        x = _solve64(pool, b, case["neumann"], 14.0 / case["pools"])
        if x is None:
            return None
        if case["kind"] == "project":
            return _gradient64(pool, x, v)
        if case["precision"] == "mixed":  # its FP64 residuals leave x on the GHOST cells too
            up = pool.parents()
            ghost = pool.rows(GHOST) & (pool.ct & INTERIOR != 0) & (_take(pool.ct, up) & INTERIOR != 0)
            x = torch.where(ghost, _take(x, up, 0.0), x)
        out.append(x)
    return out
