// Device-resident octree topology.  The reference rebuilds its adaptive grid every step with
// device kernels for the per-tile decisions and host loops for the hash-table edits (one
// cudaMalloc per new tile and host round trips in between): RefineLeafsOneStep and CoarsenStep
// (src/PoissonGrid.h:35-314), SpawnGhostTiles (src/PoissonGrid.cu:30-60), compressHost /
// syncHostAndDevice (src/HAGrid.h:491-561), CalcCellTypesFromLeafs (src/PoissonSolver.cu:7-61).
// Here everything stays on the GPU:
//   * per level two open-addressing tables of DSlot (the reference's host table, which edits go
//     to, and the device copy taken at the last sync, which the decision kernels read), with the
//     reference's hash and linear probing (src/HAAccessor.h:214-242); a tile's status word and
//     cell types live in device tile memory indexed by the slot's memory id;
//   * the per-tile decisions (refine / coarsen / delete flags, ghost candidates, cell types) are
//     data-parallel kernels;
//   * linear-probing insertion, whose result depends on the order of the requests, runs in
//     parallel with the sequential result: every request takes the first free slot of its probe
//     sequence that no earlier request takes (claim_slot);
//   * the backward-shift deletions of removeTileHost (src/HAGrid.h:409-431) run one thread per
//     cluster of occupied slots, in the reference's order inside each cluster;
//   * compaction into hash-slot order (the reference's copy_if) is one two-pass scan over the
//     tables of all levels, which also takes the synced copy.
// The host reads back one block of counters after each pass of a step (flags or candidates, then the
// compaction).  Results: the same tiles, hash slots,
// statuses and cell types as the host Topology and the reference build (tests).
#include "dtopo.hpp"

#include "common.cuh"

#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

namespace cirrus {

namespace {

constexpr int kRefineFlag = 1, kDeleteFlag = 2, kCoarsenFlag = 4;  // src/PoissonTile.h:7
constexpr int kTypeShift = 24;
constexpr int kMemMask = (1 << kTypeShift) - 1;
constexpr int kMaxMem = kMemMask + 1;  // tile memories that a slot's meta can name
// the device's counters (DevTopology::d_ctl_), read back in one copy: per level the compacted
// tiles, then the refined or deleted ones; then the appended list's length, the tile memories in
// use, and an error (level + 1 of a full table, or kDeleteErr)
constexpr int kMaxLayers = 32;
constexpr int kLevelCtl = kMaxLayers, kListCtl = 2 * kMaxLayers, kMemCtl = kListCtl + 1, kErrCtl = kListCtl + 2, kCtl = kListCtl + 3;
constexpr int kDeleteErr = 1000;
constexpr int kFirstTiles = 8192;  // tiles that the buffers hold before any grows
__constant__ int c_nb[6][3] = {{-1, 0, 0}, {1, 0, 0}, {0, -1, 0}, {0, 1, 0}, {0, 0, -1}, {0, 0, 1}};

__host__ __device__ __forceinline__ uint32_t slot_hash(int x, int y, int z, uint32_t log2) {
    uint32_t r = 0;
    r ^= (uint32_t)x * 1u;
    r ^= (uint32_t)y * 2654435761u;
    r ^= (uint32_t)z * 805459861u;
    return r & ((1u << log2) - 1u);
}
__device__ __forceinline__ int slot_type(const DSlot& s) { return s.meta < 0 ? 0 : (s.meta >> kTypeShift) & 0xff; }
__device__ __forceinline__ int slot_mem(const DSlot& s) { return s.meta & kMemMask; }

// Linear probing by one thread: the slot holding (x, y, z), or -1 (HATileAccessor::tileIdx +
// empty test).  At most `size` probes.
__device__ __forceinline__ int find_slot(const DSlot* t, uint32_t log2, int x, int y, int z) {
    const uint32_t mask = (1u << log2) - 1u;
    uint32_t k = slot_hash(x, y, z, log2);
    for (uint32_t n = 0; n <= mask; n++, k = (k + 1) & mask) {
        const DSlot s = t[k];
        if (s.meta < 0) return -1;
        if (s.x == x && s.y == y && s.z == z) return (int)k;
    }
    return -1;
}

// level target from dense per-level masks: mask[l][(x*dy + y)*dz + z] != 0, 0 outside
__device__ __forceinline__ bool mask_at(uint8_t* const* masks, const int* dims, int l, int x, int y, int z) {
    const uint8_t* m = masks[l];
    if (!m) return false;
    const int dx = dims[3 * l], dy = dims[3 * l + 1], dz = dims[3 * l + 2];
    if (x < 0 || y < 0 || z < 0 || x >= dx || y >= dy || z >= dz) return false;
    return m[((size_t)x * dy + y) * dz + z] != 0;
}

// Per-level pointers and sizes on the device, and the compacted tiles' prefix over levels: tile
// first[l] + j of the all-tiles order is arr[l][j].
struct LevelView {
    const DSlot* const* snap;  // per level
    DSlot* const* live;
    DSlot* const* arr;
    int* const* claim;
    const uint32_t* log2;
    int num_layers;
    int first[kMaxLayers + 1];
    // the level of tile q of the all-tiles order
    __device__ __forceinline__ int level_of(int q) const {
        int l = 0;
        while (q >= first[l + 1]) l++;
        return l;
    }
};

__device__ __forceinline__ const DSlot* snap_find(const LevelView& v, int l, int x, int y, int z) {
    if (l < 0 || l >= v.num_layers) return nullptr;
    const int s = find_slot(v.snap[l], v.log2[l], x, y, z);
    return s < 0 ? nullptr : &v.snap[l][s];
}
__device__ __forceinline__ DSlot* live_find(const LevelView& v, int l, int x, int y, int z) {
    if (l < 0 || l >= v.num_layers) return nullptr;
    const int s = find_slot(v.live[l], v.log2[l], x, y, z);
    return s < 0 ? nullptr : &v.live[l][s];
}

// Sum of v over the block's 256 threads, on every thread.
__device__ __forceinline__ int block_sum256(int v, int* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    int tot = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) tot += sh[k];
    __syncthreads();
    return tot;
}

// Ordered compaction of the occupied slots of all levels' tables into arr (the reference's
// thrust::copy_if keeps slot order), and the synced copy snap.  One block per chunk of kChunk
// slots, four consecutive slots per thread; chunks[b] = (level, chunk of the level, first chunk of
// the level).  Pass 1 counts, pass 2 adds up the level's preceding counts and scatters.  Bound by
// the tables' bytes (16 B read twice and written once per slot): all ten levels of the default
// hash sizes (852 k slots) take 16 us in both passes; one 1024-thread block per level walking
// its table took 134 us for each level.
constexpr int kChunk = 1024;
__global__ void __launch_bounds__(256) k_compact_count(LevelView v, const int4* __restrict__ chunks, int* counts, const int* __restrict__ ctl) {
    __shared__ int sh[8];
    if (ctl[kErrCtl]) return;  // the edits failed: the arrays stay as last synced
    const int4 c = chunks[blockIdx.x];
    const uint32_t size = 1u << v.log2[c.x], at = (uint32_t)c.y * kChunk + threadIdx.x * 4;
    const DSlot* t = v.live[c.x];
    int n = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) n += (at + e < size && t[at + e].meta >= 0) ? 1 : 0;
    n = block_sum256(n, sh);
    if (threadIdx.x == 0) counts[blockIdx.x] = n;
}
__global__ void __launch_bounds__(256) k_compact_scatter(LevelView v, const int4* __restrict__ chunks, const int* __restrict__ counts,
                                                         DSlot* const* snap, int* ctl) {
    __shared__ int sh[8];
    if (ctl[kErrCtl]) return;
    const int4 c = chunks[blockIdx.x];
    const uint32_t size = 1u << v.log2[c.x], at = (uint32_t)c.y * kChunk + threadIdx.x * 4;
    const DSlot* t = v.live[c.x];
    DSlot s[4];
    int n = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        s[e].meta = -1;
        if (at + e < size) {
            s[e] = t[at + e];
            snap[c.x][at + e] = s[e];
        }
        n += s[e].meta >= 0 ? 1 : 0;
    }
    int before = 0;
    for (int k = c.z + (int)threadIdx.x; k < (int)blockIdx.x; k += 256) before += counts[k];
    int base = block_sum256(before, sh);
    // exclusive prefix of n over the block's threads
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) sh[w] = incl;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (k < w) base += sh[k];
    int q = base + incl - n;
    DSlot* out = v.arr[c.x];
#pragma unroll
    for (int e = 0; e < 4; e++)
        if (s[e].meta >= 0) out[q++] = s[e];
    // the level's last chunk: thread 255 ends at the level's count
    if ((uint32_t)(c.y + 1) * kChunk >= size && threadIdx.x == 255) ctl[c.x] = base + incl;
}

// setTileHost (src/HAGrid.h:387-407) with blank tiles for a sequence of requests req[r] = {x, y, z,
// type} on one level, in order, by one warp (coordinates may repeat: a later request overwrites the
// type and clears the tile's memory).  Each probe step reads 32 consecutive slots; the first that is
// empty or holds the coordinates ends the probe, as in linear probing.
__global__ void __launch_bounds__(32) k_insert(DSlot* table, uint32_t log2, const int4* __restrict__ req, int n, int32_t* status,
                                               uint8_t* ctype, int* mem_count, int mem_cap, int level, int* err) {
    const int lane = threadIdx.x;
    const uint32_t size = 1u << log2, mask = size - 1u;
    int mc = *mem_count;
    for (int r = 0; r < n; r++) {
        const int4 q = req[r];
        const uint32_t h = slot_hash(q.x, q.y, q.z, log2);
        int found = -1;
        bool empty = false;
        for (uint32_t base = 0; base < size; base += 32) {
            const uint32_t k = (h + base + (uint32_t)lane) & mask;
            const DSlot s = table[k];
            const bool e = s.meta < 0, hit = !e && s.x == q.x && s.y == q.y && s.z == q.z;
            const unsigned b = __ballot_sync(0xffffffffu, (e || hit) && base + (uint32_t)lane < size);
            if (b) {
                const int first = __ffs(b) - 1;
                found = (int)((h + base + (uint32_t)first) & mask);
                empty = __shfl_sync(0xffffffffu, e, first);
                break;
            }
        }
        if (found < 0 || (empty && mc >= mem_cap)) {  // table full
            if (lane == 0) *err = level + 1;
            break;
        }
        const int mem = empty ? mc++ : slot_mem(table[found]);
        __syncwarp();
        *reinterpret_cast<uint4*>(ctype + (size_t)mem * kTileCells + lane * 16) = make_uint4(0, 0, 0, 0);
        if (lane == 0) {
            status[mem] = 0;
            DSlot s;
            s.x = q.x;
            s.y = q.y;
            s.z = q.z;
            s.meta = mem | (q.w << kTypeShift);
            table[found] = s;
        }
        __syncwarp();
    }
    if (lane == 0) *mem_count = mc;
}

// Linear-probing insertion of many distinct absent keys of one level at once, with the table that
// inserting them one by one in the order of their priorities gives.  One by one, a request takes
// the first slot of its probe sequence that is free and not taken by an earlier request.  Here a
// slot's claim is the least priority that asked for it: a request that finds its slot claimed by
// an earlier one goes on; one that claims a slot from a later one (atomicMin) leaves its thread to
// move that one on.  Claims only decrease, so a request turned away once stays turned away, and
// the claims settle on the one-by-one assignment, whatever the order of the threads.  Priorities
// are 8 * (tile of the all-tiles order) + its request, from which a displaced request's
// coordinates follow (coord).  The build of a ring512 tree and its adaptation to a moved ring insert
// some 13 k tiles: 0.18 ms in all with their parents' cell types, where one warp probing for one
// request after another took 11 ms.  No thread waits for another; a request that has been round the whole
// table reports the table full.
constexpr int kNoClaim = 0x7f7f7f7f;  // memset with 0x7f
template <class Coord>
__device__ __forceinline__ void claim_slot(const DSlot* table, int* claim, uint32_t log2, int prio, const Coord& coord, int level, int* err) {
    const uint32_t mask = (1u << log2) - 1u;
    int3 c = coord(prio);
    uint32_t h = slot_hash(c.x, c.y, c.z, log2), k = h;
    for (;;) {
        if (table[k].meta < 0) {
            const int old = atomicMin(claim + k, prio);
            if (old == kNoClaim) return;
            if (old > prio) {  // the later request goes on from here
                prio = old;
                c = coord(prio);
                h = slot_hash(c.x, c.y, c.z, log2);
            }
        }
        if (((k - h) & mask) == mask) {
            atomicMax(err, level + 1);
            return;
        }
        k = (k + 1) & mask;
    }
}
// the slot that request `prio` with these coordinates holds, or -1 (the table was full)
__device__ __forceinline__ int claimed_slot(const int* claim, uint32_t log2, int prio, int x, int y, int z) {
    const uint32_t mask = (1u << log2) - 1u;
    uint32_t k = slot_hash(x, y, z, log2);
    for (uint32_t n = 0; n <= mask; n++, k = (k + 1) & mask)
        if (claim[k] == prio) return (int)k;
    return -1;
}

// ------------------------------------------------------------------ decision kernels
// The decision kernels give a tile eight lanes, one per child or face neighbour: a probe of a hash
// table is two dependent loads, and eight of them one after another made a pass over a level 8 us
// whatever its size (5 us with eight lanes).
__device__ __forceinline__ bool any_of8(bool v) { return (__ballot_sync(0xffffffffu, v) >> (threadIdx.x & 24)) & 0xffu; }

// RefineLeafsOneStep pass 1 (src/PoissonGrid.h:50-84): LEAF tiles of level i; the refined ones (as
// tiles of the all-tiles order) are appended to list, counted in ctl[kLevelCtl + i] and ctl[kListCtl]
__global__ void __launch_bounds__(256) k_refine_leaf_flags(LevelView v, int n, int i, int dev_max, uint8_t* const* masks, const int* dims,
                                                           int32_t* status, int* list, int* ctl) {
    const int j = blockIdx.x * 32 + ((int)threadIdx.x >> 3), ci = threadIdx.x & 7;
    DSlot t;
    t.meta = -1;
    if (j < n) t = v.arr[i][j];
    const bool leaf = slot_type(t) & LEAF_T;
    bool to_refine = leaf && ci == 0 && mask_at(masks, dims, i, t.x, t.y, t.z);  // target level i + 1 > i
    if (leaf && i < dev_max) {
        const DSlot* c = snap_find(v, i + 1, t.x * 2 + (ci & 1), t.y * 2 + ((ci >> 1) & 1), t.z * 2 + ((ci >> 2) & 1));
        if (c && (slot_type(*c) & GHOST_T) && (status[slot_mem(*c)] & kRefineFlag)) to_refine = true;
    }
    to_refine = any_of8(to_refine) && i + 1 < v.num_layers;
    if (!leaf || ci != 0) return;
    int32_t& st = status[slot_mem(t)];
    st = to_refine ? (st | kRefineFlag) : (st & ~kRefineFlag);
    if (to_refine) {
        atomicAdd(ctl + kLevelCtl + i, 1);
        list[atomicAdd(ctl + kListCtl, 1)] = v.first[i] + j;
    }
}
// pass 2 (:86-102): GHOST tiles of level i take the flag of any refined LEAF neighbour
__global__ void __launch_bounds__(256) k_refine_ghost_flags(LevelView v, int n, int i, int32_t* status) {
    const int j = blockIdx.x * 32 + ((int)threadIdx.x >> 3), f = threadIdx.x & 7;
    DSlot t;
    t.meta = -1;
    if (j < n) t = v.arr[i][j];
    const bool ghost = slot_type(t) & GHOST_T;
    bool rf = false;
    if (ghost && f < 6) {
        const DSlot* nb = snap_find(v, i, t.x + c_nb[f][0], t.y + c_nb[f][1], t.z + c_nb[f][2]);
        rf = nb && (slot_type(*nb) & LEAF_T) && (status[slot_mem(*nb)] & kRefineFlag);
    }
    rf = any_of8(rf);
    if (!ghost || f != 0) return;
    int32_t& st = status[slot_mem(t)];
    st = rf ? (st | kRefineFlag) : (st & ~kRefineFlag);
}
// the host loop of the refine step (:104-129), one thread per child of the refined tiles: the
// parent's live entry becomes NONLEAF; the child's existing slot, or a claim for a new one, in the
// order (parent, child).  out[q] = (existing slot or -1, parent's tile memory).
__global__ void __launch_bounds__(256) k_refine_children(LevelView v, const int* __restrict__ list, int n, int2* out, int* ctl) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int j = list[q >> 3], ci = q & 7, i = v.level_of(j);
    const DSlot t = v.arr[i][j - v.first[i]];
    DSlot* h = live_find(v, i, t.x, t.y, t.z);
    int mem = slot_mem(t);
    if (h) {
        const int meta = h->meta;
        mem = meta & kMemMask;
        if (ci == 0) h->meta = mem | (NONLEAF_T << kTypeShift);
    }
    const int x = t.x * 2 + (ci & 1), y = t.y * 2 + ((ci >> 1) & 1), z = t.z * 2 + ((ci >> 2) & 1);
    const int s = find_slot(v.live[i + 1], v.log2[i + 1], x, y, z);
    out[q] = make_int2(s, mem);
    if (s >= 0) return;
    const DSlot* arr = v.arr[i];
    const int first = v.first[i];
    claim_slot(v.live[i + 1], v.claim[i + 1], v.log2[i + 1], 8 * j + ci,
               [arr, first](int prio) {
                   const DSlot p = arr[(prio >> 3) - first];
                   return make_int3(p.x * 2 + (prio & 1), p.y * 2 + ((prio >> 1) & 1), p.z * 2 + ((prio >> 2) & 1));
               },
               i + 1, ctl + kErrCtl);
}
// The children of level i's refined tiles list[k0 .. k0 + n / 8) into the table, one warp each: an
// existing tile keeps its memory, a new one takes the next; either receives the parent's
// childTile(child) (src/PoissonTile.h:170-191: its status and, per cell, the parent cell's type).
__global__ void __launch_bounds__(256) k_refine_place(LevelView v, const int* __restrict__ list, int k0, int n, int i,
                                                      const int2* __restrict__ found, int32_t* status, uint8_t* ctype, int* ctl) {
    const int w = blockIdx.x * 8 + ((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= n) return;
    const int q = 8 * k0 + w, j = list[q >> 3], ci = q & 7;
    const DSlot t = v.arr[i][j - v.first[i]];
    const int x = t.x * 2 + (ci & 1), y = t.y * 2 + ((ci >> 1) & 1), z = t.z * 2 + ((ci >> 2) & 1);
    DSlot* table = v.live[i + 1];
    const int2 f = found[q];
    int s = f.x, mem = 0;
    if (lane == 0) {
        if (s >= 0) {
            mem = slot_mem(table[s]);
        } else {
            s = claimed_slot(v.claim[i + 1], v.log2[i + 1], 8 * j + ci, x, y, z);
            if (s >= 0) mem = atomicAdd(ctl + kMemCtl, 1);
        }
    }
    s = __shfl_sync(0xffffffffu, s, 0);
    mem = __shfl_sync(0xffffffffu, mem, 0);
    if (s < 0) return;
    const int sm = f.y, ox = ci & 1, oy = (ci >> 1) & 1, oz = (ci >> 2) & 1;
    uint8_t bytes[16];
#pragma unroll
    for (int e = 0; e < 16; e++) {
        const int c = lane * 16 + e, a = c >> 6, b = (c >> 3) & 7, cc = c & 7;
        bytes[e] = ctype[(size_t)sm * kTileCells + ((((ox * 8 + a) >> 1) << 6) | (((oy * 8 + b) >> 1) << 3) | ((oz * 8 + cc) >> 1))];
    }
    uint4 u;
    memcpy(&u, bytes, 16);
    *reinterpret_cast<uint4*>(ctype + (size_t)mem * kTileCells + lane * 16) = u;
    if (lane == 0) {
        status[mem] = status[sm];
        DSlot d;
        d.x = x;
        d.y = y;
        d.z = z;
        d.meta = mem | (LEAF_T << kTypeShift);
        table[s] = d;
        if (f.x < 0) v.claim[i + 1][s] = kNoClaim;
    }
}
// SpawnGhostTiles candidates (src/PoissonGrid.cu:36-56): for every LEAF|NONLEAF tile of the
// compacted arrays above level 0 and each face neighbour whose parent is a LEAF of the live level
// l-1 table and which the live table lacks, a claim in the order (tile, face).  Several tiles may
// ask for one GHOST tile: the first in that order does, the others (which the reference finds
// existing by then) drop out.
__global__ void __launch_bounds__(256) k_ghost_candidates(LevelView v, int n, int* list, int* ctl) {
    const int q = v.first[1] * 8 + blockIdx.x * blockDim.x + threadIdx.x;  // 8 * tile + face
    const int j = q >> 3, f = q & 7;
    if (j >= n || f >= 6) return;
    const int l = v.level_of(j), first = v.first[l];
    const DSlot* arr = v.arr[l];
    const DSlot t = arr[j - first];
    if (!(slot_type(t) & (LEAF_T | NONLEAF_T))) return;
    const int nx = t.x + c_nb[f][0], ny = t.y + c_nb[f][1], nz = t.z + c_nb[f][2];
    const DSlot* p = live_find(v, l - 1, nx >> 1, ny >> 1, nz >> 1);
    if (!p || !(slot_type(*p) & LEAF_T)) return;
    if (find_slot(v.live[l], v.log2[l], nx, ny, nz) >= 0) return;
    // the all-tiles order inside a level is the order of the synced table's slots
    const int own = find_slot(v.snap[l], v.log2[l], t.x, t.y, t.z);
    for (int g = 0; g < 6; g++) {  // the tile on whose face g the GHOST tile lies
        if (g == f) continue;
        const int s = find_slot(v.snap[l], v.log2[l], nx - c_nb[g][0], ny - c_nb[g][1], nz - c_nb[g][2]);
        if (s >= 0 && s < own && (slot_type(v.snap[l][s]) & (LEAF_T | NONLEAF_T))) return;
    }
    list[atomicAdd(ctl + kListCtl, 1)] = q;
    claim_slot(v.live[l], v.claim[l], v.log2[l], q,
               [arr, first](int prio) {
                   const DSlot o = arr[(prio >> 3) - first];
                   const int g = prio & 7;
                   return make_int3(o.x + c_nb[g][0], o.y + c_nb[g][1], o.z + c_nb[g][2]);
               },
               l, ctl + kErrCtl);
}
// the claimed GHOST tiles into the tables with blank memory, one warp each
__global__ void __launch_bounds__(256) k_ghost_place(LevelView v, const int* __restrict__ list, int n, int32_t* status, uint8_t* ctype, int* ctl) {
    const int w = blockIdx.x * 8 + ((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= n) return;
    const int q = list[w], j = q >> 3, f = q & 7, l = v.level_of(j);
    const DSlot t = v.arr[l][j - v.first[l]];
    DSlot d;
    d.x = t.x + c_nb[f][0];
    d.y = t.y + c_nb[f][1];
    d.z = t.z + c_nb[f][2];
    int s = -1, mem = 0;
    if (lane == 0) {
        s = claimed_slot(v.claim[l], v.log2[l], q, d.x, d.y, d.z);
        if (s >= 0) mem = atomicAdd(ctl + kMemCtl, 1);
    }
    s = __shfl_sync(0xffffffffu, s, 0);
    mem = __shfl_sync(0xffffffffu, mem, 0);
    if (s < 0) return;
    *reinterpret_cast<uint4*>(ctype + (size_t)mem * kTileCells + lane * 16) = make_uint4(0, 0, 0, 0);
    if (lane == 0) {
        status[mem] = 0;
        d.meta = mem | (GHOST_T << kTypeShift);
        v.live[l][s] = d;
        v.claim[l][s] = kNoClaim;
    }
}

// CoarsenStep flags (src/PoissonGrid.h:172-276)
__device__ __forceinline__ void set_mask(int32_t& st, int m, bool on) { st = on ? (st | m) : (st & ~m); }
__global__ void __launch_bounds__(256) k_coarsen_nonleaf(LevelView v, int n, int l, int32_t* status) {
    const int j = blockIdx.x * 32 + ((int)threadIdx.x >> 3), ci = threadIdx.x & 7;
    DSlot t;
    t.meta = -1;
    if (j < n) t = v.arr[l][j];
    const bool nonleaf = slot_type(t) & NONLEAF_T;
    bool keep = false;
    if (nonleaf) {
        const DSlot* c = snap_find(v, l + 1, t.x * 2 + (ci & 1), t.y * 2 + ((ci >> 1) & 1), t.z * 2 + ((ci >> 2) & 1));
        keep = !c || !(slot_type(*c) & LEAF_T) || !(status[slot_mem(*c)] & kDeleteFlag);
    }
    keep = any_of8(keep);
    if (!nonleaf || ci != 0) return;
    int32_t& st = status[slot_mem(t)];
    set_mask(st, kCoarsenFlag, !keep);
    set_mask(st, kDeleteFlag, false);
}
__global__ void __launch_bounds__(256) k_coarsen_leaf(LevelView v, int n, int l, uint8_t* const* masks, const int* dims, int32_t* status) {
    const int j = blockIdx.x * 32 + ((int)threadIdx.x >> 3), f = threadIdx.x & 7;
    DSlot t;
    t.meta = -1;
    if (j < n) t = v.arr[l][j];
    const bool leaf = slot_type(t) & LEAF_T;
    bool keep = false;
    if (leaf && f < 6) {
        const DSlot* nb = snap_find(v, l, t.x + c_nb[f][0], t.y + c_nb[f][1], t.z + c_nb[f][2]);
        keep = nb && (slot_type(*nb) & NONLEAF_T) && !(status[slot_mem(*nb)] & kCoarsenFlag);
    }
    keep = any_of8(keep);
    if (!leaf || f != 0) return;
    int32_t& st = status[slot_mem(t)];
    set_mask(st, kCoarsenFlag, false);
    set_mask(st, kDeleteFlag, !keep && mask_at(masks, dims, l, t.x, t.y, t.z));  // target level l - 1 < l
}
__global__ void k_coarsen_down(LevelView v, int n, int l, int32_t* status) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const DSlot t = v.arr[l][j];
    if (!(slot_type(t) & (LEAF_T | GHOST_T))) return;
    bool to_delete = false;
    const DSlot* p = snap_find(v, l - 1, t.x >> 1, t.y >> 1, t.z >> 1);
    if (p && (status[slot_mem(*p)] & kCoarsenFlag)) to_delete = true;
    int32_t& st = status[slot_mem(t)];
    set_mask(st, kDeleteFlag, to_delete);
    if (to_delete) set_mask(st, kCoarsenFlag, true);
}
__global__ void __launch_bounds__(256) k_coarsen_ghost(LevelView v, int n, int l, int32_t* status) {
    const int j = blockIdx.x * 32 + ((int)threadIdx.x >> 3), f = threadIdx.x & 7;
    DSlot t;
    t.meta = -1;
    if (j < n) t = v.arr[l][j];
    const bool ghost = slot_type(t) & GHOST_T;
    bool keep = false;
    if (ghost && f < 6) {
        const DSlot* nb = snap_find(v, l, t.x + c_nb[f][0], t.y + c_nb[f][1], t.z + c_nb[f][2]);
        keep = nb && (slot_type(*nb) & LEAF_T) && !(status[slot_mem(*nb)] & kDeleteFlag);
    }
    keep = any_of8(keep);
    if (ghost && f == 0 && !keep) status[slot_mem(t)] |= kDeleteFlag;
}
// CoarsenStep's table edits (src/PoissonGrid.h:280-305): in all-tiles order a tile flagged for
// deletion is removed (removeTileHost's backward shift, src/HAGrid.h:409-431), one flagged for
// coarsening becomes LEAF.  An edit only touches its own cluster, the run of occupied slots between
// two empty ones, so the clusters are edited in parallel, each by one thread in order (ring512's
// coarsening: 86 us in both passes, 1.3 ms by one thread).  This pass
// finds, before any edit, the clusters that have one: leaders[k] = (level, first slot, slots).
__device__ __forceinline__ int coarsen_op(const DSlot& t, const int32_t* status) {
    if (t.meta < 0) return 0;
    const int32_t st = status[slot_mem(t)];
    return (st & kDeleteFlag) ? 1 : (st & kCoarsenFlag) ? 2 : 0;
}
__global__ void __launch_bounds__(256) k_coarsen_clusters(LevelView v, const int4* __restrict__ chunks, const int32_t* __restrict__ status,
                                                          int4* leaders, int* ctl) {
    const int4 c = chunks[blockIdx.x];
    const int l = c.x;
    const uint32_t size = 1u << v.log2[l], mask = size - 1u;
    const DSlot* live = v.live[l];
    for (uint32_t at = (uint32_t)c.y * kChunk + threadIdx.x, e = 0; e < 4 && at < size; e++, at += 256) {
        if (live[at].meta < 0) continue;
        bool lead = live[(at - 1) & mask].meta < 0;
        if (at == 0 && !lead) {  // slot 0 leads a table without an empty slot
            uint32_t k = mask;
            while (k > 0 && live[k].meta >= 0) k--;
            lead = k == 0;
        }
        if (!lead) continue;
        uint32_t len = 0;
        bool any = false;
        while (len < size && live[(at + len) & mask].meta >= 0) {
            any = any || coarsen_op(v.snap[l][(at + len) & mask], status) != 0;
            len++;
        }
        if (any) leaders[atomicAdd(ctl + kListCtl, 1)] = make_int4(l, (int)at, (int)len, 0);
    }
}
__global__ void __launch_bounds__(64) k_coarsen_edit(LevelView v, const int4* __restrict__ leaders, const int32_t* __restrict__ status, int* ctl) {
    const int n = ctl[kListCtl];
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int4 c = leaders[q];
        const int l = c.x;
        const uint32_t log2 = v.log2[l], size = 1u << log2, mask = size - 1u;
        DSlot* table = v.live[l];
        // slots in order: the part of a cluster that runs past the table's end comes first
        const uint32_t wrapped = (uint32_t)c.y + (uint32_t)c.z > size ? (uint32_t)c.y + (uint32_t)c.z - size : 0u;
        for (uint32_t e = 0; e < (uint32_t)c.z; e++) {
            const DSlot t = v.snap[l][e < wrapped ? e : (uint32_t)c.y + e - wrapped];
            const int op = coarsen_op(t, status);
            if (op == 0) continue;
            if (op == 1) atomicAdd(ctl + kLevelCtl + l, 1);
            const int s = find_slot(table, log2, t.x, t.y, t.z);
            if (s < 0) continue;
            if (op == 2) {
                table[s].meta = slot_mem(table[s]) | (LEAF_T << kTypeShift);
                continue;
            }
            uint32_t i = (uint32_t)s, j = i;
            for (uint32_t guard = 0; guard <= mask; guard++) {
                j = (j + 1) & mask;
                const DSlot sj = table[j];
                if (sj.meta < 0) break;
                const uint32_t k = slot_hash(sj.x, sj.y, sj.z, log2);
                if ((j > i && (k <= i || k > j)) || (j < i && (k <= i && k > j))) {
                    const DSlot si = table[i];
                    table[i] = sj;
                    table[j] = si;
                    i = j;
                }
                if (guard == mask) atomicMax(ctl + kErrCtl, kDeleteErr);
            }
            table[i].meta = -1;
        }
    }
}

// CalcCellTypesFromLeafs (src/PoissonSolver.cu:7-61).  Step 1, one level at a time from fine to
// coarse, one block per NONLEAF tile: a cell is DIRICHLET if any LEAF|NONLEAF child cell is, else
// INTERIOR if any is, else NEUMANN.
__global__ void __launch_bounds__(128) k_celltypes_nonleaf(LevelView v, int n, int l, uint8_t* ctype) {
    __shared__ int child_mem[8];
    const int j = blockIdx.x;
    if (j >= n) return;
    const DSlot t = v.arr[l][j];
    if (!(slot_type(t) & NONLEAF_T)) return;
    if (threadIdx.x < 8) {
        const int ci = threadIdx.x;
        const DSlot* c = snap_find(v, l + 1, t.x * 2 + (ci & 1), t.y * 2 + ((ci >> 1) & 1), t.z * 2 + ((ci >> 2) & 1));
        child_mem[ci] = (c && (slot_type(*c) & (LEAF_T | NONLEAF_T))) ? slot_mem(*c) : -1;
    }
    __syncthreads();
    uint8_t* out = ctype + (size_t)slot_mem(t) * kTileCells;
    for (int o = threadIdx.x; o < kTileCells; o += blockDim.x) {
        const int i = o >> 6, jj = (o >> 3) & 7, k = o & 7;
        int dcnt = 0, icnt = 0;
        for (int c = 0; c < 8; c++) {
            const int gx = (i * 2 + (c & 1)), gy = (jj * 2 + ((c >> 1) & 1)), gz = (k * 2 + ((c >> 2) & 1));
            // the child tile holding fine cell (gx, gy, gz) of this tile's 16^3 refinement
            const int cm = child_mem[(gx >> 3) | ((gy >> 3) << 1) | ((gz >> 3) << 2)];
            if (cm < 0) continue;
            const uint8_t tt = ctype[(size_t)cm * kTileCells + ((gx & 7) << 6) + ((gy & 7) << 3) + (gz & 7)];
            if (tt & DIRICHLET_C) dcnt++;
            else if (tt & INTERIOR_C) icnt++;
        }
        out[o] = dcnt > 0 ? DIRICHLET_C : (icnt > 0 ? INTERIOR_C : NEUMANN_C);
    }
}
// Step 2: a GHOST cell takes its parent cell's type, DIRICHLET without a parent tile.
__global__ void __launch_bounds__(128) k_celltypes_ghost(LevelView v, int n, int l, uint8_t* ctype) {
    const int j = blockIdx.x;
    if (j >= n) return;
    const DSlot t = v.arr[l][j];
    if (!(slot_type(t) & GHOST_T)) return;
    const DSlot* p = snap_find(v, l - 1, t.x >> 1, t.y >> 1, t.z >> 1);
    const int pm = p ? slot_mem(*p) : -1;
    uint8_t* out = ctype + (size_t)slot_mem(t) * kTileCells;
    const int ox = t.x & 1, oy = t.y & 1, oz = t.z & 1;
    for (int o = threadIdx.x; o < kTileCells; o += blockDim.x) {
        const int i = o >> 6, jj = (o >> 3) & 7, k = o & 7;
        const int pc = (((ox * 8 + i) >> 1) << 6) | (((oy * 8 + jj) >> 1) << 3) | ((oz * 8 + k) >> 1);
        out[o] = pm >= 0 ? ctype[(size_t)pm * kTileCells + pc] : DIRICHLET_C;
    }
}

// exports, one thread or block per tile of the all-tiles order
__global__ void k_tile_rows(LevelView v, int n, int32_t* out5) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int l = v.level_of(q);
    const DSlot t = v.arr[l][q - v.first[l]];
    int32_t* o = out5 + (size_t)5 * q;
    o[0] = l;
    o[1] = t.x;
    o[2] = t.y;
    o[3] = t.z;
    o[4] = slot_type(t);
}
__global__ void k_slots_of(LevelView v, int n, int32_t* slot) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int l = v.level_of(q);
    const DSlot t = v.arr[l][q - v.first[l]];
    slot[q] = find_slot(v.live[l], v.log2[l], t.x, t.y, t.z);
}
__global__ void __launch_bounds__(128) k_copy_types(LevelView v, int n, uint8_t* ctype, uint8_t* host_order, int to_mem) {
    const int q = blockIdx.x * 4 + ((int)threadIdx.x >> 5), lane = threadIdx.x & 31;  // one warp per tile
    if (q >= n) return;
    const int l = v.level_of(q);
    uint4* m = reinterpret_cast<uint4*>(ctype + (size_t)slot_mem(v.arr[l][q - v.first[l]]) * kTileCells) + lane;
    uint4* a = reinterpret_cast<uint4*>(host_order + (size_t)q * kTileCells) + lane;
    if (to_mem) *m = *a;
    else *a = *m;
}
__global__ void k_gather_status(LevelView v, int n, const int32_t* __restrict__ status, int32_t* out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int l = v.level_of(q);
    out[q] = status[slot_mem(v.arr[l][q - v.first[l]])];
}

// Tile q of the all-tiles order gets memory q in the compacted arrays and in both tables, which hold
// the same tiles in the same slots.
__global__ void k_renumber(LevelView v, int n, DSlot* const* snap) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int l = v.level_of(q);
    DSlot& t = v.arr[l][q - v.first[l]];
    const int meta = q | (slot_type(t) << kTypeShift), s = find_slot(v.live[l], v.log2[l], t.x, t.y, t.z);
    t.meta = meta;
    if (s < 0) return;
    v.live[l][s].meta = meta;
    snap[l][s].meta = meta;
}

inline int blocks(int n, int b = 256) { return std::max(1, (n + b - 1) / b); }

#define DT_CK(x)                                                           \
    do {                                                                   \
        cudaError_t e_ = (x);                                              \
        if (e_ != cudaSuccess) {                                           \
            last_error = std::string(#x ": ") + cudaGetErrorString(e_);    \
            return e_ == cudaErrorMemoryAllocation ? 3 : 2;                \
        }                                                                  \
    } while (0)

}  // namespace

// The last destroyed topology's allocation is kept for the next one of the same size in its context: a
// simulator that rebuilds its grid makes and destroys one every time, and an allocation of this size
// and its release took 1.1 ms of a 5 ms build on one machine, 3 to 8 ms on another.  At most one block
// of at most kKeepBytes is kept; it is given back when another replaces it or an allocation of the
// library finds device memory used up (device_malloc).  An address outlives its context -- after a device reset another allocation may
// lie there -- so the block goes by its context's id, which the driver gives no second time, and only
// blocks of a device's primary context are kept, whose end that id tells.
namespace {
constexpr size_t kKeepBytes = 128u << 20;
struct KeptBlock {
    std::mutex lock;
    void* p = nullptr;
    size_t bytes = 0;
    int device = -1;
    unsigned long long context = 0;
};
KeptBlock& kept() {
    static KeptBlock* k = new KeptBlock;  // not destroyed: objects may outlive static destruction
    return *k;
}

struct Driver {
    CUresult (*ctx_id)(CUcontext, unsigned long long*) = nullptr;
    CUresult (*primary_state)(CUdevice, unsigned int*, int*) = nullptr;
    CUresult (*primary_retain)(CUcontext*, CUdevice) = nullptr;
    CUresult (*primary_release)(CUdevice) = nullptr;
    Driver() {
        auto get = [](const char* name, auto& f) {
            void* p = nullptr;
            cudaDriverEntryPointQueryResult q;
            if (cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
                return false;
            f = reinterpret_cast<std::decay_t<decltype(f)>>(p);
            return true;
        };
        ok = get("cuCtxGetId", ctx_id) && get("cuDevicePrimaryCtxGetState", primary_state) &&
             get("cuDevicePrimaryCtxRetain", primary_retain) && get("cuDevicePrimaryCtxRelease", primary_release);
    }
    bool ok = false;
};
const Driver& driver() {
    static const Driver d;
    return d;
}
// The id of the device's primary context, 0 while it has none.
unsigned long long primary_context(int device) {
    const Driver& d = driver();
    unsigned int flags = 0;
    int active = 0;
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (!d.ok || d.primary_state(device, &flags, &active) != CUDA_SUCCESS || !active || d.primary_retain(&c, device) != CUDA_SUCCESS) return 0;
    if (d.ctx_id(c, &id) != CUDA_SUCCESS) id = 0;
    d.primary_release(device);
    return id;
}
// The current device's context if the calling thread uses its primary one, else 0.
unsigned long long current_context(int device) {
    const Driver& d = driver();
    unsigned long long id = 0;
    if (!d.ok || d.ctx_id(nullptr, &id) != CUDA_SUCCESS) return 0;
    return id == primary_context(device) ? id : 0;
}

// Frees the kept block, or forgets it when its context is gone.
void drop_kept(KeptBlock& k) {
    if (k.p && k.context == primary_context(k.device)) cudaFree(k.p);
    k.p = nullptr;
}
void* take_kept(size_t bytes, unsigned long long context) {
    KeptBlock& k = kept();
    std::lock_guard<std::mutex> l(k.lock);
    if (!k.p || k.bytes != bytes || context == 0 || k.context != context) return nullptr;
    void* p = k.p;
    k.p = nullptr;
    return p;
}
// Takes over the block p that a topology made in `context` leaves.
void keep(void* p, size_t bytes, int device, unsigned long long context) {
    // (nothing of the object's is in flight once the stream all its work is on has drained)
    if (bytes > kKeepBytes || context == 0 || current_context(device) != context || cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
        cudaFree(p);
        return;
    }
    KeptBlock& k = kept();
    std::lock_guard<std::mutex> l(k.lock);
    drop_kept(k);
    k.p = p;
    k.bytes = bytes;
    k.device = device;
    k.context = context;
}
}  // namespace

cudaError_t device_malloc_bytes(void** p, size_t bytes) {
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    {
        KeptBlock& k = kept();
        std::lock_guard<std::mutex> l(k.lock);
        if (!k.p) return e;
        drop_kept(k);
    }
    cudaGetLastError();
    return cudaMalloc(p, bytes);
}

// Per-level tables and everything else of a fixed size live in one allocation (three tables of
// DSlot and the insertion claims per level, the compaction's chunk list and counts, the pointer
// tables), with first sizes of the buffers that grow: a grid of kFirstTiles tiles allocates once (an
// allocation and its release cost 0.2-0.5 ms each, as much as a whole refinement).
DevTopology::DevTopology(int num_layers, const uint32_t* log2_hash, double h0)
    : num_layers_(num_layers), h0_(h0), log2_(log2_hash, log2_hash + num_layers) {
    live_.assign(num_layers, nullptr);
    snap_.assign(num_layers, nullptr);
    arr_.assign(num_layers, nullptr);
    count_.assign(num_layers, 0);
    std::vector<int*> claim(num_layers, nullptr);
    std::vector<int4> chunks;
    size_t slots = 0;
    for (int l = 0; l < num_layers; l++) {
        const size_t size = (size_t)1 << log2_[l];
        const int first = (int)chunks.size();
        for (size_t c = 0; c * kChunk < size; c++) chunks.push_back(make_int4(l, (int)c, first, 0));
        slots += size;
    }
    n_chunks_ = (int)chunks.size();
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t tables = up(sizeof(DSlot) * slots), claims = up(sizeof(int) * slots), ch = up(sizeof(int4) * chunks.size()),
                 cc = up(sizeof(int) * chunks.size()), ptrs = up(sizeof(void*) * num_layers), small = up(sizeof(int) * 4 * kMaxLayers);
    unsigned char* base = nullptr;
    // lists hold up to 24 bytes per tile, the children's slots 64, masks 128, cell types 512
    const size_t list = up(16 * kFirstTiles), types = (size_t)kFirstTiles * kTileCells, st = up(sizeof(int32_t) * kFirstTiles);
    const size_t bytes = 3 * tables + claims + ch + cc + 5 * ptrs + 3 * small + 14 * list + 2 * types + st;
    cudaGetDevice(&device_);
    cudaFree(nullptr);  // the thread's context exists and is current from here
    context_ = current_context(device_);
    base = (unsigned char*)take_kept(bytes, context_);
    if (!base && device_malloc(&base, bytes) != cudaSuccess) {
        last_error = "device topology: allocation failed";
        return;
    }
    d_base_ = base;
    base_bytes_ = bytes;
    auto take = [&](size_t b) {
        unsigned char* p = base;
        base += b;
        return p;
    };
    DSlot *live = (DSlot*)take(tables), *snap = (DSlot*)take(tables), *arr = (DSlot*)take(tables);
    int* cl = (int*)take(claims);
    d_chunks_ = (int4*)take(ch);
    d_chunk_count_ = (int*)take(cc);
    d_live_ = (DSlot**)take(ptrs);
    d_snap_ = (DSlot**)take(ptrs);
    d_arr_ = (DSlot**)take(ptrs);
    d_claim_ = (int**)take(ptrs);
    d_masks_ = (uint8_t**)take(ptrs);
    d_log2_ = (uint32_t*)take(small);
    d_mask_dims_ = (int*)take(small);
    d_ctl_ = (int*)take(small);
    static_assert(kCtl <= 4 * kMaxLayers, "counters fit their block");
    auto buffer = [&](Buffer& b, size_t n) {
        b.p = take(n);
        b.cap = n;
    };
    buffer(scratch_, 2 * list);
    buffer(mask_buf_, 8 * list);
    buffer(found_, 4 * list);
    buffer(export_, types);
    ctype_ = take(types);
    status_ = (int32_t*)take(st);
    mem_cap_ = kFirstTiles;
    d_claims_ = cl;
    claim_slots_ = slots;
    size_t off = 0;
    for (int l = 0; l < num_layers; l++) {
        live_[l] = live + off;
        snap_[l] = snap + off;
        arr_[l] = arr + off;
        claim[l] = cl + off;
        off += (size_t)1 << log2_[l];
    }
    bool ok = cudaMemset(live, 0xff, 2 * tables) == cudaSuccess;  // live and snap: meta = -1, empty
    ok = ok && cudaMemset(cl, 0x7f, claims) == cudaSuccess && cudaMemset(d_ctl_, 0, small) == cudaSuccess;
    auto put = [&](void* d, const void* h, size_t b) { ok = ok && cudaMemcpy(d, h, b, cudaMemcpyHostToDevice) == cudaSuccess; };
    put(d_chunks_, chunks.data(), sizeof(int4) * chunks.size());
    put(d_live_, live_.data(), sizeof(void*) * num_layers);
    put(d_snap_, snap_.data(), sizeof(void*) * num_layers);
    put(d_arr_, arr_.data(), sizeof(void*) * num_layers);
    put(d_claim_, claim.data(), sizeof(void*) * num_layers);
    put(d_log2_, log2_.data(), sizeof(uint32_t) * num_layers);
    if (!ok) last_error = "device topology: allocation failed";
}

DevTopology::~DevTopology() {
    for (Buffer* b : {&mask_buf_, &scratch_, &found_, &export_})
        if (b->owned) cudaFree(b->p);
    if (mem_owned_) {
        cudaFree(status_);
        cudaFree(ctype_);
    }
    if (d_base_) keep(d_base_, base_bytes_, device_, context_);
}

int DevTopology::num_tiles() const {
    int n = 0;
    for (int c : count_) n += c;
    return n;
}

// the kernels' view of the tables and of the compacted tiles' order
static LevelView level_view(DSlot** snap, DSlot** live, DSlot** arr, int** claim, uint32_t* log2, const std::vector<int>& count) {
    LevelView v;
    v.snap = snap;
    v.live = live;
    v.arr = arr;
    v.claim = claim;
    v.log2 = log2;
    v.num_layers = (int)count.size();
    int n = 0;
    for (int l = 0; l <= kMaxLayers; l++) {
        v.first[l] = n;
        if (l < (int)count.size()) n += count[l];
    }
    return v;
}
#define DT_VIEW level_view(d_snap_, d_live_, d_arr_, d_claim_, d_log2_, count_)

// A deleted tile's memory goes to no other tile until the memories are renumbered: instead of growing
// where that frees half of them, and where a slot's meta could not name the next ones.
int DevTopology::ensure_mem(int extra) {
    if ((long long)mem_count_ + extra <= mem_cap_) return 0;
    const long long held = (long long)num_tiles() + extra;
    if (!stale_ && (2 * held <= mem_cap_ || (long long)mem_count_ + extra > kMaxMem)) {
        const int rc = renumber_mem();
        if (rc) return rc;
        if (held <= mem_cap_) return 0;
    }
    if ((long long)mem_count_ + extra > kMaxMem) {
        last_error = "device topology: more than 2^24 tile memories";
        return 4;
    }
    const int cap = std::min(std::max(mem_count_ + extra, mem_cap_ * 2), kMaxMem);
    int32_t* st = nullptr;
    uint8_t* ct = nullptr;
    DT_CK(device_malloc(&st, sizeof(int32_t) * cap));
    const cudaError_t e = device_malloc(&ct, (size_t)cap * kTileCells);
    if (e != cudaSuccess) {
        cudaFree(st);
        DT_CK(e);
    }
    if (mem_count_ > 0) {
        DT_CK(cudaMemcpy(st, status_, sizeof(int32_t) * mem_count_, cudaMemcpyDeviceToDevice));
        DT_CK(cudaMemcpy(ct, ctype_, (size_t)mem_count_ * kTileCells, cudaMemcpyDeviceToDevice));
    }
    if (mem_owned_) {
        cudaFree(status_);
        cudaFree(ctype_);
    }
    status_ = st;
    ctype_ = ct;
    mem_cap_ = cap;
    mem_owned_ = true;
    return 0;
}

// Statuses and cell types into the all-tiles order, by way of the exports' buffer.
int DevTopology::renumber_mem() {
    const int n = num_tiles();
    if (n > 0) {
        std::lock_guard<std::mutex> lock(export_lock_);
        const size_t types = (size_t)n * kTileCells, words = sizeof(int32_t) * (size_t)n;
        const int rc = grow(&export_, types + words);
        if (rc) return rc;
        uint8_t* to = (uint8_t*)export_.p;
        const LevelView v = DT_VIEW;
        k_copy_types<<<blocks(n, 4), 128>>>(v, n, ctype_, to, 0);
        k_gather_status<<<blocks(n), 256>>>(v, n, status_, (int32_t*)(to + types));
        k_renumber<<<blocks(n), 256>>>(v, n, d_snap_);
        DT_CK(cudaMemcpyAsync(ctype_, to, types, cudaMemcpyDeviceToDevice));
        DT_CK(cudaMemcpyAsync(status_, to + types, words, cudaMemcpyDeviceToDevice));
    }
    DT_CK(cudaMemcpy(d_ctl_ + kMemCtl, &n, sizeof(int), cudaMemcpyHostToDevice));
    mem_count_ = n;
    return 0;
}

// At least `bytes` in b (contents are not kept).
int DevTopology::grow(Buffer* b, size_t bytes) const {
    if (bytes <= b->cap) return 0;
    if (b->owned) cudaFree(b->p);
    b->p = nullptr;
    b->cap = 0;
    b->owned = true;
    const size_t want = bytes + bytes / 2;
    const cudaError_t e = device_malloc(&b->p, want);
    if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? 3 : 2;
    b->cap = want;
    return 0;
}

// The counters of the last step; the list's and the per-level ones are cleared for the next.
int DevTopology::read_ctl(int* ctl) {
    DT_CK(cudaMemcpy(ctl, d_ctl_, sizeof(int) * kCtl, cudaMemcpyDeviceToHost));
    DT_CK(cudaMemsetAsync(d_ctl_ + kLevelCtl, 0, sizeof(int) * (kMaxLayers + 1)));
    mem_count_ = ctl[kMemCtl];
    if (ctl[kErrCtl]) {
        last_error = ctl[kErrCtl] == kDeleteErr ? "device topology: deletion did not terminate"
                                                : "hash table full at level " + std::to_string(ctl[kErrCtl] - 1);
        cudaMemset(d_ctl_ + kErrCtl, 0, sizeof(int));
        cudaMemset(d_claims_, 0x7f, sizeof(int) * claim_slots_);
        return 4;
    }
    return 0;
}

int DevTopology::set_tiles(int level, const int32_t* xyz, const uint8_t* types, int n) {
    if (level < 0 || level >= num_layers_ || n < 0) {
        last_error = "level out of range";
        return 1;
    }
    if (n == 0) return 0;
    std::vector<int4> req(n);
    for (int i = 0; i < n; i++) req[i] = make_int4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], types[i]);
    int rc = grow(&scratch_, sizeof(int4) * n);
    if (!rc) rc = ensure_mem(n);
    if (rc) return rc;
    DT_CK(cudaMemcpy(scratch_.p, req.data(), sizeof(int4) * n, cudaMemcpyHostToDevice));
    k_insert<<<1, 32>>>(live_[level], log2_[level], (const int4*)scratch_.p, n, status_, ctype_, d_ctl_ + kMemCtl, mem_cap_, level,
                        d_ctl_ + kErrCtl);
    stale_ = true;
    int ctl[kCtl];
    return read_ctl(ctl);
}

int DevTopology::compress_and_sync() {
    const LevelView v = DT_VIEW;
    k_compact_count<<<n_chunks_, 256>>>(v, d_chunks_, d_chunk_count_, d_ctl_);
    k_compact_scatter<<<n_chunks_, 256>>>(v, d_chunks_, d_chunk_count_, d_snap_, d_ctl_);
    DT_CK(cudaGetLastError());
    int ctl[kCtl];
    const int rc = read_ctl(ctl);
    if (rc) return rc;
    max_level_ = -1;
    for (int l = 0; l < num_layers_; l++) {
        count_[l] = ctl[l];
        if (count_[l] > 0) max_level_ = l;
    }
    stale_ = false;
    return 0;
}

int DevTopology::spawn_ghost_tiles() {
    const LevelView v = DT_VIEW;
    const int n = num_tiles(), above = n - v.first[1];
    int m = 0;
    if (above > 0) {
        int rc = grow(&scratch_, sizeof(int) * 6 * (size_t)above);
        if (rc) return rc;
        k_ghost_candidates<<<blocks(8 * above), 256>>>(v, n, (int*)scratch_.p, d_ctl_);
        int ctl[kCtl];
        rc = read_ctl(ctl);
        if (rc) return rc;
        m = ctl[kListCtl];
    }
    if (m > 0) {
        const int rc = ensure_mem(m);
        if (rc) {
            cudaMemset(d_claims_, 0x7f, sizeof(int) * claim_slots_);
            return rc;
        }
        stale_ = true;
        k_ghost_place<<<blocks(m, 8), 256>>>(v, (const int*)scratch_.p, m, status_, ctype_, d_ctl_);
    }
    return stale_ ? compress_and_sync() : 0;  // (nothing edited: the tables are as last synced)
}

int DevTopology::upload_masks(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims) {
    std::vector<uint8_t*> ptrs(num_layers_, nullptr);
    std::vector<size_t> off(num_layers_ + 1, 0);
    for (int l = 0; l < num_layers_; l++) {
        const size_t n = l < (int)masks.size() && masks[l] ? (size_t)dims[3 * l] * dims[3 * l + 1] * dims[3 * l + 2] : 0;
        off[l + 1] = off[l] + (n + 15) / 16 * 16;
    }
    const int rc = grow(&mask_buf_, std::max<size_t>(off[num_layers_], 1));
    if (rc) return rc;
    for (int l = 0; l < num_layers_; l++) {
        if (off[l + 1] == off[l]) continue;
        ptrs[l] = (uint8_t*)mask_buf_.p + off[l];
        DT_CK(cudaMemcpy(ptrs[l], masks[l], (size_t)dims[3 * l] * dims[3 * l + 1] * dims[3 * l + 2], cudaMemcpyHostToDevice));
    }
    DT_CK(cudaMemcpy(d_masks_, ptrs.data(), sizeof(uint8_t*) * num_layers_, cudaMemcpyHostToDevice));
    DT_CK(cudaMemcpy(d_mask_dims_, dims.data(), sizeof(int) * 3 * num_layers_, cudaMemcpyHostToDevice));
    return 0;
}

// All levels' flags first, finest first (a level's LEAF flags read the flags of the GHOST tiles one
// level finer); then the refined tiles, listed level by level in that order, become NONLEAF and
// their children are inserted.  The insertions follow in the same order of levels, so a child that
// overwrites a tile does so after that tile's own children were made from it.
int DevTopology::refine_step(std::vector<int>* counts) {
    const LevelView v = DT_VIEW;
    const int n = num_tiles();
    std::vector<int> cnt(num_layers_, 0);
    int m = 0;
    if (n > 0) {
        int rc = grow(&scratch_, sizeof(int) * (size_t)n);
        if (rc) return rc;
        for (int i = max_level_; i >= 0; i--) {
            if (count_[i] == 0) continue;
            k_refine_leaf_flags<<<blocks(count_[i], 32), 256>>>(v, count_[i], i, max_level_, d_masks_, d_mask_dims_, status_, (int*)scratch_.p, d_ctl_);
            if (i > 0) k_refine_ghost_flags<<<blocks(count_[i], 32), 256>>>(v, count_[i], i, status_);
        }
        int ctl[kCtl];
        rc = read_ctl(ctl);
        if (rc) return rc;
        m = ctl[kListCtl];
        for (int l = 0; l < num_layers_; l++) cnt[l] = ctl[kLevelCtl + l];
    }
    if (m > 0) {
        int rc = ensure_mem(8 * m);
        if (!rc) rc = grow(&found_, sizeof(int2) * 8 * (size_t)m);
        if (rc) return rc;
        const int* list = (const int*)scratch_.p;
        stale_ = true;
        k_refine_children<<<blocks(8 * m), 256>>>(v, list, 8 * m, (int2*)found_.p, d_ctl_);
        for (int i = max_level_, k0 = 0; i >= 0; k0 += cnt[i], i--)
            if (cnt[i] > 0) k_refine_place<<<blocks(8 * cnt[i], 8), 256>>>(v, list, k0, 8 * cnt[i], i, (const int2*)found_.p, status_, ctype_, d_ctl_);
    }
    if (counts) *counts = cnt;
    return stale_ ? compress_and_sync() : 0;
}

int DevTopology::refine_leafs_one_step(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims, std::vector<int>* counts) {
    const int rc = upload_masks(masks, dims);
    return rc ? rc : refine_step(counts);
}

int DevTopology::iterative_refine(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims) {
    // src/PoissonGrid.h:316-326
    int rc = upload_masks(masks, dims);
    if (rc) return rc;
    for (int guard = 0; guard < 64; guard++) {
        std::vector<int> c;
        rc = refine_step(&c);
        if (rc) return rc;
        rc = spawn_ghost_tiles();
        if (rc) return rc;
        int tot = 0;
        for (int x : c) tot += x;
        if (tot == 0) return 0;
    }
    last_error = "iterative refine did not settle";
    return 4;
}

int DevTopology::coarsen_step(const std::vector<const uint8_t*>& masks, const std::vector<int>& dims, std::vector<int>* deleted) {
    int rc = upload_masks(masks, dims);
    if (rc) return rc;
    const LevelView v = DT_VIEW;
    const int n_all = num_tiles();
    for (int l = num_layers_ - 1; l >= 0; l--) {
        const int n = count_[l];
        if (n == 0) continue;
        k_coarsen_nonleaf<<<blocks(n, 32), 256>>>(v, n, l, status_);
        k_coarsen_leaf<<<blocks(n, 32), 256>>>(v, n, l, d_masks_, d_mask_dims_, status_);
    }
    for (int l = 0; l < num_layers_; l++) {
        const int n = count_[l];
        if (n == 0) continue;
        k_coarsen_down<<<blocks(n), 256>>>(v, n, l, status_);
        k_coarsen_ghost<<<blocks(n, 32), 256>>>(v, n, l, status_);
    }
    std::vector<int> del(num_layers_, 0);
    if (n_all > 0) {
        rc = grow(&scratch_, sizeof(int4) * (size_t)n_all);  // a cluster has a tile at least
        if (rc) return rc;
        k_coarsen_clusters<<<n_chunks_, 256>>>(v, d_chunks_, status_, (int4*)scratch_.p, d_ctl_);
        stale_ = true;
        k_coarsen_edit<<<blocks(n_all, 64), 64>>>(v, (const int4*)scratch_.p, status_, d_ctl_);
        int ctl[kCtl];
        rc = read_ctl(ctl);
        if (rc) return rc;
        for (int l = 0; l < num_layers_; l++) del[l] = ctl[kLevelCtl + l];
    }
    if (deleted) *deleted = del;
    return compress_and_sync();
}

int DevTopology::calc_cell_types_from_leafs() {
    const LevelView v = DT_VIEW;
    for (int l = num_layers_ - 1; l >= 0; l--)
        if (count_[l] > 0) k_celltypes_nonleaf<<<count_[l], 128>>>(v, count_[l], l, ctype_);
    for (int l = 0; l < num_layers_; l++)
        if (count_[l] > 0) k_celltypes_ghost<<<count_[l], 128>>>(v, count_[l], l, ctype_);
    DT_CK(cudaDeviceSynchronize());
    return 0;
}

// Exports through one buffer that only grows; the exports are const and may be called from several
// threads, so they take turns at it.
template <class Launch>
int DevTopology::export_with(size_t bytes, void* host, Launch&& launch) const {
    std::lock_guard<std::mutex> lock(export_lock_);
    const int rc = grow(&export_, bytes);
    if (rc) return rc;
    launch(export_.p);
    return cudaMemcpy(host, export_.p, bytes, cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : 2;
}

int DevTopology::tiles(int32_t* out5) const {
    const int n = num_tiles();
    if (n == 0) return 0;
    return export_with(sizeof(int32_t) * 5 * n, out5, [&](void* d) { k_tile_rows<<<blocks(n), 256>>>(DT_VIEW, n, (int32_t*)d); });
}

int DevTopology::hash_slots(int32_t* out) const {
    const int n = num_tiles();
    if (n == 0) return 0;
    return export_with(sizeof(int32_t) * n, out, [&](void* d) { k_slots_of<<<blocks(n), 256>>>(DT_VIEW, n, (int32_t*)d); });
}

int DevTopology::cell_types(uint8_t* out) const {
    const int n = num_tiles();
    if (n == 0) return 0;
    return export_with((size_t)n * kTileCells, out, [&](void* d) { k_copy_types<<<blocks(n, 4), 128>>>(DT_VIEW, n, ctype_, (uint8_t*)d, 0); });
}

int DevTopology::set_cell_types(const uint8_t* host_ct) {
    const int n = num_tiles();
    if (n == 0) return 0;
    std::lock_guard<std::mutex> lock(export_lock_);
    const int rc = grow(&export_, (size_t)n * kTileCells);
    if (rc) return rc;
    DT_CK(cudaMemcpy(export_.p, host_ct, (size_t)n * kTileCells, cudaMemcpyHostToDevice));
    k_copy_types<<<blocks(n, 4), 128>>>(DT_VIEW, n, ctype_, (uint8_t*)export_.p, 1);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
}

int DevTopology::statuses(int32_t* out) const {
    const int n = num_tiles();
    if (n == 0) return 0;
    return export_with(sizeof(int32_t) * n, out, [&](void* d) { k_gather_status<<<blocks(n), 256>>>(DT_VIEW, n, status_, (int32_t*)d); });
}

}  // namespace cirrus
