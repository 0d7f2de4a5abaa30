"""The device topology on tables that are nearly full, where requests collide, clusters of occupied
slots run long and wrap around the table's end: parallel insertion against the host topology (one
request after another), and the clusters' deletions against CoarsenStep restated in Python."""
from __future__ import annotations

import numpy as np
import pytest

from cirrus_b200 import CirrusError, DeviceTopology, Topology, workloads as W

pytestmark = pytest.mark.gpu

FACES = ((-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1))
# log2 hash sizes that hold the workload's tiles per level with little or nothing to spare
TIGHT = {"uniform32_small": (1, 3, 6), "sphere64_small": (1, 3, 6, 9), "ring64_small": (1, 4, 7, 8), "sphere256": (1, 3, 6, 9, 11, 12)}


def build(w, log2):
    d = DeviceTopology(w.h0, log2)
    d.set_tiles(0, np.array(w.roots, dtype=np.int32), W.LEAF)
    d.compress()
    d.spawn_ghost_tiles()
    d.iterative_refine(w.masks[:len(log2)])
    return d


@pytest.mark.parametrize("name", sorted(TIGHT))
def test_tight_tables_equal_host(name):
    w, log2 = W.make(name), TIGHT[name]
    d = build(w, log2)
    t = Topology(w.h0, log2)
    for r in w.roots:
        t.set_tile(0, r, W.LEAF)
    t.compress()
    t.spawn_ghost_tiles()
    t.iterative_refine(masks=w.masks[:len(log2)])
    assert np.array_equal(d.tiles(), t.tiles())
    assert np.array_equal(d.hash_slots(), t.hash_slots())


def test_full_table_is_reported():
    w = W.make("sphere64_small")
    with pytest.raises(CirrusError):
        build(w, (1, 3, 6, 8))  # level 3 holds 400 tiles


def test_step_after_a_full_table_syncs_its_edits():
    """A refinement that found its table full has edited the live tables: a next step that adds nothing
    still compacts them, as an explicit compaction does."""
    d = DeviceTopology(0.125, (1, 2, 3))
    d.set_tiles(0, np.array([[0, 0, 0]], dtype=np.int32), W.LEAF)
    d.compress()
    with pytest.raises(CirrusError):
        d.refine_leafs_one_step([np.ones((1, 1, 1), dtype=np.uint8), None, None])  # eight children, four slots
    d.spawn_ghost_tiles()
    tiles = d.tiles()
    d.compress()
    assert np.array_equal(tiles, d.tiles())


def coarsen_reference(tiles, slots, log2, masks):
    """CoarsenStep on the tables given by tiles and slots: (tiles and slots after, deleted per level)."""
    size = [1 << b for b in log2]
    table = [[None] * s for s in size]
    kind, order = [{} for _ in log2], [[] for _ in log2]
    for (l, x, y, z, ty), s in zip(tiles.tolist(), slots.tolist()):
        table[l][s] = (x, y, z)
        kind[l][(x, y, z)] = ty
        order[l].append((x, y, z))
    coarsen, delete = [set() for _ in log2], [set() for _ in log2]

    def near(c):
        return [(c[0] + a, c[1] + b, c[2] + e) for a, b, e in FACES]

    for l in reversed(range(len(log2))):
        for c in [c for c in order[l] if kind[l][c] == W.NONLEAF]:
            kids = [(2 * c[0] + (i & 1), 2 * c[1] + (i >> 1 & 1), 2 * c[2] + (i >> 2)) for i in range(8)]
            if all(kind[l + 1].get(k) == W.LEAF and k in delete[l + 1] for k in kids):
                coarsen[l].add(c)
        for c in [c for c in order[l] if kind[l][c] == W.LEAF]:
            m = masks[l]
            if m is not None and m[c] and not any(kind[l].get(k) == W.NONLEAF and k not in coarsen[l] for k in near(c)):
                delete[l].add(c)
    for l in range(len(log2)):
        for c in [c for c in order[l] if kind[l][c] in (W.LEAF, W.GHOST)]:
            gone = l > 0 and (c[0] >> 1, c[1] >> 1, c[2] >> 1) in coarsen[l - 1]
            (delete[l].add if gone else delete[l].discard)(c)
            if gone:
                coarsen[l].add(c)
        for c in [c for c in order[l] if kind[l][c] == W.GHOST]:
            if not any(kind[l].get(k) == W.LEAF and k not in delete[l] for k in near(c)):
                delete[l].add(c)
    count = [0] * len(log2)
    for l in range(len(log2)):
        mask = size[l] - 1

        def home(c):
            return (c[0] ^ (c[1] * 2654435761) ^ (c[2] * 805459861)) & 0xFFFFFFFF & mask

        for c in order[l]:
            if c in delete[l]:
                count[l] += 1
                i = table[l].index(c)
                j = i
                while True:
                    j = (j + 1) & mask
                    if table[l][j] is None:
                        break
                    k = home(table[l][j])
                    if (j > i and (k <= i or k > j)) or (j < i and k <= i and k > j):
                        table[l][i], table[l][j] = table[l][j], table[l][i]
                        i = j
                table[l][i] = None
            elif c in coarsen[l]:
                kind[l][c] = W.LEAF
    out = [(l, *c, kind[l][c], s) for l in range(len(log2)) for s, c in enumerate(table[l]) if c is not None]
    return np.array([o[:5] for o in out], dtype=np.int32), np.array([o[5] for o in out], dtype=np.int32), count


@pytest.mark.parametrize("name", ["sphere64_small", "ring64_small", "sphere256"])
def test_coarsening_tight_tables(name):
    w, log2 = W.make(name), TIGHT[name]
    if name != "sphere256":
        log2 = log2[:-1] + (log2[-1] + 1,)  # a deletion needs an empty slot to stop at
    d = build(w, log2)
    fine = max(l for l in range(len(log2)) if w.masks[l - 1] is not None)
    for part in (2, 1):  # half of the domain, then the rest
        tiles, slots = d.tiles(), d.hash_slots()
        masks = [None] * len(log2)
        masks[fine] = np.zeros([e << fine for e in w.root_extent], dtype=np.uint8)
        masks[fine][: masks[fine].shape[0] // part] = 1
        want_tiles, want_slots, want = coarsen_reference(tiles, slots, log2, masks)
        assert d.coarsen_step(masks) == want and sum(want) > 0
        assert np.array_equal(d.tiles(), want_tiles)
        assert np.array_equal(d.hash_slots(), want_slots)
        d.spawn_ghost_tiles()


def test_topologies_one_after_another_and_at_once():
    """A destroyed topology's memory serves the next one: builds of different trees in turn, two alive
    at a time and from several threads, each equal to the host's."""
    from concurrent.futures import ThreadPoolExecutor

    names = ["sphere64_small", "ring64_small", "uniform32_small"]
    host = {}
    for n in names:
        w = W.make(n)
        t = Topology(w.h0, w.log2_hash)
        for r in w.roots:
            t.set_tile(0, r, W.LEAF)
        t.compress()
        t.spawn_ghost_tiles()
        t.iterative_refine(masks=w.masks)
        host[n] = t.tiles()

    def one(n):
        w = W.make(n)
        a = build(w, w.log2_hash)
        b = build(w, w.log2_hash)
        assert np.array_equal(a.tiles(), host[n])
        del a
        assert np.array_equal(b.tiles(), host[n])

    for n in names * 2:
        one(n)
    with ThreadPoolExecutor(4) as ex:
        list(ex.map(one, names * 4))


AFTER_RESET = """
import ctypes as C, sys
sys.path.insert(0, {root!r})
import numpy as np
from cirrus_b200 import DeviceTopology, Topology, workloads as W

w = W.make("sphere64_small")
t = Topology(w.h0, w.log2_hash)
for r in w.roots:
    t.set_tile(0, r, W.LEAF)
t.compress()
t.spawn_ghost_tiles()
t.iterative_refine(masks=w.masks)

def build():
    d = DeviceTopology(w.h0, w.log2_hash)
    d.set_tiles(0, np.array(w.roots, dtype=np.int32), W.LEAF)
    d.compress()
    d.spawn_ghost_tiles()
    d.iterative_refine(w.masks)
    assert np.array_equal(d.tiles(), t.tiles())

cu = C.CDLL("libcuda.so.1")
for turn in range(2):
    build()  # leaves its block behind
    assert cu.cuDevicePrimaryCtxReset_v2(0) == 0
    ctx = C.c_void_p()
    assert cu.cuDevicePrimaryCtxRetain(C.byref(ctx), 0) == 0 and cu.cuCtxSetCurrent(ctx) == 0
    others = []  # other allocations where the block lay
    for mb in (64, 32, 16, 8, 4, 2, 64, 64):
        p = C.c_uint64()
        assert cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(mb << 20)) == 0
        assert cu.cuMemsetD8_v2(p, C.c_ubyte(0xa5), C.c_size_t(mb << 20)) == 0
        others.append((p, mb << 20))
    build()
    for p, n in others:
        h = np.empty(n, dtype=np.uint8)
        assert cu.cuMemcpyDtoH_v2(C.c_void_p(h.ctypes.data), p, C.c_size_t(n)) == 0
        assert (h == 0xa5).all()
        assert cu.cuMemFree_v2(p) == 0
print("ok")
"""


def test_a_kept_block_ends_with_its_context():
    """After a device reset another allocation may have the address of the block that a destroyed
    topology left; the next topology leaves it alone.  (A child process: the reset ends its context.)"""
    import subprocess
    import sys
    from pathlib import Path

    root = str(Path(__file__).resolve().parents[1])
    r = subprocess.run([sys.executable, "-c", AFTER_RESET.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr


def check_own_memory(d, seed):
    """No two tiles share their memory: every tile gives back the cell types it was given."""
    ct = np.random.default_rng(seed).integers(0, 8, (d.num_tiles, 512), dtype=np.uint8)
    d.set_cell_types(ct)
    assert np.array_equal(d.cell_types(), ct)


def test_adapting_past_the_nameable_memories():
    """Refined and coarsened back until 2^24 tile memories have been given out (262144 a time): the
    deleted tiles' are used again, and tables, statuses and cell types stay those of the first time."""
    d = DeviceTopology(0.125, (1, 4, 7, 10, 13, 16, 19))
    d.set_tiles(0, np.array([[0, 0, 0]], dtype=np.int32), W.LEAF)
    d.compress()
    d.iterative_refine([np.ones((1 << l,) * 3, dtype=np.uint8) for l in range(5)] + [None, None])
    check_own_memory(d, 1)
    up = [None] * 5 + [np.ones((32,) * 3, dtype=np.uint8), None]
    down = [None] * 6 + [np.ones((64,) * 3, dtype=np.uint8)]
    first, most = None, 0
    while most <= 1 << 24:
        assert d.refine_leafs_one_step(up)[5] == 32768
        assert d.coarsen_step(down)[6] == 262144
        most += 262144
        if first is None:
            first = d.tiles(), d.hash_slots(), d.statuses(), d.cell_types()
    for a, b in zip(first, (d.tiles(), d.hash_slots(), d.statuses(), d.cell_types())):
        assert np.array_equal(a, b)
    d.refine_leafs_one_step(up)
    check_own_memory(d, 2)


def test_adapting_a_tree_with_ghost_tiles_many_times():
    """Past 8192 tile memories in all, a few hundred tiles at a time: the tables after each coarsening
    are CoarsenStep's, and every tile has its own memory."""
    w, log2 = W.make("ring64_small"), TIGHT["ring64_small"]
    log2 = log2[:-1] + (log2[-1] + 1,)
    d = build(w, log2)
    fine = max(l for l in range(len(log2)) if w.masks[l - 1] is not None)
    masks = [None] * len(log2)
    masks[fine] = np.ones([e << fine for e in w.root_extent], dtype=np.uint8)
    given = d.num_tiles
    while given < 3 * 8192:
        want_tiles, want_slots, want = coarsen_reference(d.tiles(), d.hash_slots(), log2, masks)
        assert d.coarsen_step(masks) == want
        assert np.array_equal(d.tiles(), want_tiles) and np.array_equal(d.hash_slots(), want_slots)
        d.spawn_ghost_tiles()
        n = d.num_tiles
        d.iterative_refine(w.masks[:len(log2)])
        assert d.num_tiles > n
        given += d.num_tiles - n
        check_own_memory(d, given)


def test_a_kept_block_is_given_back_when_memory_runs_out(built_cache):
    """With the device's memory filled up to a few MB, preparing the AMG coefficients (54 MB) gets the
    room that a destroyed topology's block took."""
    import torch

    from cirrus_b200 import AMGSolver, DeviceGrid

    small = DeviceGrid(built_cache("sphere64_small").topology)
    AMGSolver().prepare_types_and_coeffs(small)  # the kernels are loaded before memory runs out
    b = built_cache("sphere256")
    g = DeviceGrid(b.topology)
    need = 17 * 512 * g.num_tiles
    build(W.make("sphere64_small"), (16,) * 6 + (18,) * 4)  # leaves more than that behind
    fill, size = [], 1 << 36
    torch.cuda.synchronize()
    try:
        while size >= 2 << 20:
            try:
                fill.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                size >>= 1
        assert torch.cuda.mem_get_info()[0] < need
        AMGSolver().prepare_types_and_coeffs(g)
    finally:
        fill.clear()
        torch.cuda.empty_cache()
