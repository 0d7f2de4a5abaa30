// The AMG variant of the preconditioner (AMGSolver, src/AMGSolver.h, src/AMGSolver.cu): explicit
// per-cell face coefficients, coarse-level coefficients and cell types formed from the children
// (Galerkin-style), Gauss-Seidel smoothing and residuals on those coefficients, and the same PCG
// as GMGSolver::solve around the V-cycle.  In the reference the class is dead code at its only
// call site (src/FluidEuler.h:592-593, commented out) and its file does not build in this
// environment (VTK and Eigen includes), so the arithmetic here is the CPU restatement's
// (oracle/cirrus_oracle.cpp, AMG section), checked bit for bit on the GPU, with no reference
// output to pin it.
//
// Storage: four FP32 planes of n*512 (off-diagonal coefficient of each cell's x-, y-, z- face,
// then the diagonal) and a byte plane of AMG cell types (the grid's cell types with GHOST cells
// re-derived from their parents and NONLEAF cells rewritten by the coarsening), allocated on the
// first prepare.  The kernels take one 128-thread CTA per tile, thread t owning the cells
// 4t..4t+3 (column (t >> 4, (t >> 1) & 7), k = 4 (t & 1) .. +3); the coarsest level's sweeps run
// as one CTA per instance looping over its tiles (k_amg_gs_sequence).  Tiles of finished
// instances are skipped (per-instance scalars S), so the V-cycle runs inside batched solves too.
#include "kernels.cuh"
#include "solver_internal.hpp"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace cirrus {

namespace {

constexpr uint8_t kTypedCell = INTERIOR_C | DIRICHLET_C | NEUMANN_C;

__device__ __forceinline__ int cell_of(int i, int j, int k) { return (i << 6) | (j << 3) | k; }

// GHOST cells take their parent cell's type, DIRICHLET without a parent (src/AMGSolver.cu:118-133);
// every other cell keeps the grid's type.
__global__ void __launch_bounds__(128) k_amg_types(Topo tp, int n, uint8_t* __restrict__ act) {
    const int tile = blockIdx.x;
    if (tile >= n) return;
    const TileMeta m = tp.meta[tile];
    const bool ghost = meta_type(m.packed) & GHOST_T;
    const int oct = meta_octant(m.packed);
    for (int c = threadIdx.x; c < kTileCells; c += blockDim.x) {
        uint8_t v = tp.ctype[(size_t)tile * kTileCells + c];
        if (ghost) {
            const int i = c >> 6, j = (c >> 3) & 7, k = c & 7;
            v = m.parent < 0 ? DIRICHLET_C
                             : tp.ctype[(size_t)m.parent * kTileCells +
                                        cell_of((oct & 1) * 4 + (i >> 1), ((oct >> 1) & 1) * 4 + (j >> 1), ((oct >> 2) & 1) * 4 + (k >> 1))];
        }
        act[(size_t)tile * kTileCells + c] = v;
    }
}

// CalculateAMGCoefficients on LEAF|GHOST tiles (src/AMGSolver.cu:16-108): per cell and face in
// (axis, -/+) order the coefficient 1/h^2 (LEAF-LEAF) or (1/(1.5h))/h (LEAF-GHOST), 0 for other
// pairs or next to a NEUMANN cell, times h^3; an absent neighbour tile counts as a DIRICHLET cell
// of the cell's own tile type.  The diagonal sums the six; the off-diagonal of a lower face is
// minus its coefficient when the neighbour is INTERIOR.  Non-INTERIOR cells store zeros.
// Products and sums rounded one by one (no fused multiply-adds).
__global__ void __launch_bounds__(128) k_amg_coeffs(Topo tp, const int* __restrict__ list, int n, const uint8_t* __restrict__ act,
                                                    float* __restrict__ C, size_t plane) {
    const int q = blockIdx.x;
    if (q >= n) return;
    const int tile = list[q];
    const TileMeta m = tp.meta[tile];
    const int tt0 = meta_type(m.packed);
    int ntt[6];
#pragma unroll
    for (int f = 0; f < 6; f++) ntt[f] = m.nb[f] >= 0 ? meta_type(tp.meta[m.nb[f]].packed) : tt0;
    const float h = tile_level_const(tp, tile, meta_level(m.packed)).h;
    const float oh = __fdiv_rn(1.f, h), ogh = __fdiv_rn(1.f, __fmul_rn(1.5f, h));
    const size_t base = (size_t)tile * kTileCells;
    for (int c = threadIdx.x; c < kTileCells; c += blockDim.x) {
        const int ijk[3] = {c >> 6, (c >> 3) & 7, c & 7};
        const uint8_t ct0 = act[base + c];
        float diag = 0.f, off[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int axis = 0; axis < 3; axis++)
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const int stride = axis == 0 ? 64 : axis == 1 ? 8 : 1;
                const bool inside = s == 0 ? ijk[axis] > 0 : ijk[axis] < 7;
                const int f = 2 * axis + s;
                int tt1 = tt0;
                uint8_t ct1 = DIRICHLET_C;
                if (inside) {
                    ct1 = act[base + c + (s == 0 ? -stride : stride)];
                } else if (m.nb[f] >= 0) {
                    tt1 = ntt[f];
                    ct1 = act[(size_t)m.nb[f] * kTileCells + c + (s == 0 ? 7 * stride : -7 * stride)];
                }
                const bool both = (tt0 & LEAF_T) && (tt1 & LEAF_T);
                const bool olog = ((tt0 & LEAF_T) && (tt1 & GHOST_T)) || ((tt0 & GHOST_T) && (tt1 & LEAF_T));
                const float odh = both ? oh : olog ? ogh : 0.f;
                const bool nm = (ct0 & NEUMANN_C) || (ct1 & NEUMANN_C);
                float cf = nm ? 0.f : __fdiv_rn(odh, h);
                cf = __fmul_rn(__fmul_rn(__fmul_rn(cf, h), h), h);
                if (s == 0 && ct1 == INTERIOR_C) off[axis] = -cf;
                diag = __fadd_rn(diag, cf);
            }
        const bool interior = ct0 == INTERIOR_C;
#pragma unroll
        for (int a = 0; a < 3; a++) C[a * plane + base + c] = interior ? off[a] : 0.f;
        C[3 * plane + base + c] = interior ? diag : 0.f;
    }
}

// CoarsenTypesAndAMGCoeffs step 3 on the LEAF and NONLEAF tiles of one level, after the finer
// level (src/AMGSolver.cu:138-203): per cell over its 2x2x2 children in (ci, cj, ck) order the
// sum of their diagonals and INTERIOR count, then the lower-face off-diagonals of the children on
// the cell's lower faces summed per axis and twice those of the interior faces added to the
// diagonal.  NONLEAF: type INTERIOR if any child is, else DIRICHLET; coefficients = sums times
// one_over_alpha.  LEAF with a GHOST child tile: sums added to its own coefficients.
__global__ void __launch_bounds__(128) k_amg_coarsen(Topo tp, const int* __restrict__ child, int first, int count, uint8_t* __restrict__ act,
                                                     float* __restrict__ C, size_t plane, float one_over_alpha) {
    const int q = blockIdx.x;
    if (q >= count) return;
    const int tile = first + q;
    const int tt = meta_type(tp.meta[tile].packed);
    if (tt != LEAF_T && tt != NONLEAF_T) return;
    const size_t base = (size_t)tile * kTileCells;
    for (int c = threadIdx.x; c < kTileCells; c += blockDim.x) {
        const int i = c >> 6, j = (c >> 3) & 7, k = c & 7;
        const int ch = child[(size_t)tile * 8 + ((i >> 2) | ((j >> 2) << 1) | ((k >> 2) << 2))];
        bool ghost_child = false;
        float cod[3][8];
        float diag_sum = 0.f;
        int interior_cnt = 0;
        if (ch >= 0) {
            ghost_child = meta_type(tp.meta[ch].packed) == GHOST_T;
            const size_t cb = (size_t)ch * kTileCells;
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const int cid = cell_of(2 * (i & 3) + (b >> 2), 2 * (j & 3) + ((b >> 1) & 1), 2 * (k & 3) + (b & 1));
                diag_sum = __fadd_rn(diag_sum, C[3 * plane + cb + cid]);
                interior_cnt += act[cb + cid] == INTERIOR_C ? 1 : 0;
#pragma unroll
                for (int a = 0; a < 3; a++) cod[a][b] = C[a * plane + cb + cid];
            }
        } else {
#pragma unroll
            for (int b = 0; b < 8; b++)
#pragma unroll
                for (int a = 0; a < 3; a++) cod[a][b] = 0.f;
        }
        float offs[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const int ci = b >> 2, cj = (b >> 1) & 1, ck = b & 1;
            if (ci == 0) offs[0] = __fadd_rn(offs[0], cod[0][b]);
            else diag_sum = __fadd_rn(diag_sum, __fmul_rn(2.f, cod[0][b]));
            if (cj == 0) offs[1] = __fadd_rn(offs[1], cod[1][b]);
            else diag_sum = __fadd_rn(diag_sum, __fmul_rn(2.f, cod[1][b]));
            if (ck == 0) offs[2] = __fadd_rn(offs[2], cod[2][b]);
            else diag_sum = __fadd_rn(diag_sum, __fmul_rn(2.f, cod[2][b]));
        }
        if (tt == NONLEAF_T) {
            act[base + c] = interior_cnt > 0 ? INTERIOR_C : DIRICHLET_C;
#pragma unroll
            for (int a = 0; a < 3; a++) C[a * plane + base + c] = __fmul_rn(offs[a], one_over_alpha);
            C[3 * plane + base + c] = __fmul_rn(diag_sum, one_over_alpha);
        } else if (ghost_child) {
#pragma unroll
            for (int a = 0; a < 3; a++) C[a * plane + base + c] = __fadd_rn(C[a * plane + base + c], offs[a]);
            C[3 * plane + base + c] = __fadd_rn(C[3 * plane + base + c], diag_sum);
        }
    }
}

// AMGLaplacianTileData::negativeLapSameLevel (src/AMGSolver.cu:231-250) of cell (i, j, k) of a
// staged tile: x0 * diag, then per face in (axis, -/+) order the off-diagonal stored at the face's
// upper cell times the neighbour's x, fused into the sum.  A lower face's coefficient is the
// cell's own; an upper face's is the next cell's, across the tile face the neighbour tile's first
// cell (0 when that tile is absent, as is its x in the staged halo).
__device__ __forceinline__ float amg_lap(const TileShared<float>& sh, const float* __restrict__ C, size_t plane, size_t base,
                                         const TileMeta& m, int i, int j, int k) {
    const int c = cell_of(i, j, k);
    float sum = __fmul_rn(sh.xs[c], C[3 * plane + base + c]);
    const int ijk[3] = {i, j, k};
#pragma unroll
    for (int axis = 0; axis < 3; axis++) {
        const int stride = axis == 0 ? 64 : axis == 1 ? 8 : 1;
        // halo slot of the cell's column on an axis face: x faces [j*8 + k], y faces [i*8 + k], z faces [i*8 + j]
        const int hs = axis == 0 ? j * 8 + k : axis == 1 ? i * 8 + k : i * 8 + j;
        const float xm = ijk[axis] > 0 ? sh.xs[c - stride] : sh.hx[(2 * axis) * 64 + hs];
        sum = fmaf(C[axis * plane + base + c], xm, sum);
        float xp, cp;
        if (ijk[axis] < 7) {
            xp = sh.xs[c + stride];
            cp = C[axis * plane + base + c + stride];
        } else {
            xp = sh.hx[(2 * axis + 1) * 64 + hs];
            const int nb = m.nb[2 * axis + 1];
            cp = nb >= 0 ? C[axis * plane + (size_t)nb * kTileCells + c - 7 * stride] : 0.f;
        }
        sum = fmaf(cp, xp, sum);
    }
    return sum;
}

// NegativeLaplacianAndGaussSeidelSameLevel128Kernel (src/AMGSolver.cu:540-578) on the LEAF|NONLEAF
// tiles of one level: cells of colour (i+j+k)%2 == color get x + (b - A x)/D where INTERIOR, x + 0
// elsewhere.
// The colour update of thread t's four cells of a staged tile (see k_amg_gs).
__device__ __forceinline__ void amg_gs_cells(const TileShared<float>& sh, const float* __restrict__ C, size_t plane, int tile, const TileMeta& m,
                                             int t, float* X, const float* __restrict__ RHS, const uint8_t* __restrict__ act, int color) {
    const TileIdx ix(t);
    const size_t base = (size_t)tile * kTileCells;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int k = ix.k0 + e;
        if (((ix.i + ix.j + k) & 1) != color) continue;
        const int c = cell_of(ix.i, ix.j, k);
        float delta = 0.f;
        if (act[base + c] & INTERIOR_C) {
            const float ax = amg_lap(sh, C, plane, base, m, ix.i, ix.j, k);
            delta = __fdiv_rn(RHS[base + c] - ax, C[3 * plane + base + c]);
        }
        X[base + c] = sh.xs[c] + delta;
    }
}

__global__ void __launch_bounds__(128) k_amg_gs(Topo tp, const int* __restrict__ list, int n, float* X, const float* __restrict__ RHS,
                                                const uint8_t* __restrict__ act, const float* __restrict__ C, size_t plane, int color,
                                                const Scalars* __restrict__ S) {
    pdl_entry_for(RHS, act, C, S);
    __shared__ TileShared<float> sh;
    const int q = blockIdx.x, t = threadIdx.x;
    const int tile = q < n ? list[q] : 0;
    const bool active = q < n && !tile_done(tp, S, tile);
    TileMeta m;
    if (active) {
        m = tp.meta[tile];
        stage_tile<float>(X, tile, m, t, sh);
    }
    __syncthreads();
    if (!active) return;
    amg_gs_cells(sh, C, plane, tile, m, t, X, RHS, act, color);
}

// A sequence of colour sweeps (bit s of `colors` = the colour of sweep s) over one level's
// LEAF|NONLEAF tiles, one CTA per instance: CTA i takes the list entries ranges[i] = (first, count)
// -- one instance's tiles, coupled to no other instance's -- in rounds of blockDim/128 tiles, and
// a __syncthreads makes each round's global writes visible to the next round's halo loads.  A
// colour's cells never neighbour each other, so updating a sweep's tiles round by round gives
// the bits of one launch per sweep.
__global__ void __launch_bounds__(1024) k_amg_gs_sequence(Topo tp, const int* __restrict__ list, const int2* __restrict__ ranges,
                                                          float* X, const float* __restrict__ RHS, const uint8_t* __restrict__ act,
                                                          const float* __restrict__ C, size_t plane, uint32_t colors, int nsweeps,
                                                          const Scalars* __restrict__ S) {
    pdl_entry_for(RHS, act, C, S);
    __shared__ TileShared<float> sh[8];
    const int2 r = ranges[blockIdx.x];
    const int groups = blockDim.x >> 7;
    const int g = threadIdx.x >> 7, t = threadIdx.x & 127;
    for (int s = 0; s < nsweeps; s++) {
        const int color = (colors >> s) & 1;
        for (int base = 0; base < r.y; base += groups) {
            const int q = base + g;
            const int tile = q < r.y ? list[r.x + q] : 0;
            const bool active = q < r.y && !tile_done(tp, S, tile);
            TileMeta m;
            if (active) {
                m = tp.meta[tile];
                stage_tile<float>(X, tile, m, t, sh[g]);
            }
            __syncthreads();
            if (active) amg_gs_cells(sh[g], C, plane, tile, m, t, X, RHS, act, color);
            __syncthreads();
        }
    }
}

// The downstroke's residual (src/AMGSolver.cu:640-643): on every tile of the level,
// TMP = RHS - A x on INTERIOR cells, 0 elsewhere.
__global__ void __launch_bounds__(128) k_amg_residual(Topo tp, int first, int n, const float* __restrict__ X, const float* __restrict__ RHS,
                                                      float* __restrict__ TMP, const uint8_t* __restrict__ act, const float* __restrict__ C,
                                                      size_t plane, const Scalars* __restrict__ S) {
    pdl_entry_for(X, RHS, act, C, S);
    __shared__ TileShared<float> sh;
    const int q = blockIdx.x, t = threadIdx.x;
    const int tile = first + (q < n ? q : 0);
    const bool active = q < n && !tile_done(tp, S, tile);
    TileMeta m;
    if (active) {
        m = tp.meta[tile];
        stage_tile<float>(X, tile, m, t, sh);
    }
    __syncthreads();
    if (!active) return;
    const TileIdx ix(t);
    const size_t base = (size_t)tile * kTileCells;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int c = cell_of(ix.i, ix.j, ix.k0 + e);
        TMP[base + c] = act[base + c] == INTERIOR_C ? RHS[base + c] - amg_lap(sh, C, plane, base, m, ix.i, ix.j, ix.k0 + e) : 0.f;
    }
}

// Restriction to the coarser level (src/AMGSolver.cu:646-652) on every tile of that level:
// NONLEAF: Restrict (src/PoissonSolver.cu:292-319) -- 0 on non-INTERIOR cells, then, if the
// tile's first child tile exists, the children's INTERIOR residuals summed in child-index order
// (x fastest) times one_over_alpha; LEAF: Copy of F + AccumulateToParents of the GHOST children's
// residuals (src/PoissonGrid.cu:721-755, typed cells, added with coefficient 1); GHOST: Fill 0.
__global__ void __launch_bounds__(128) k_amg_restrict(Topo tp, const int* __restrict__ child, int first, int n, const float* __restrict__ F,
                                                      const float* __restrict__ TMP, float* __restrict__ RHS, const uint8_t* __restrict__ act,
                                                      float one_over_alpha, const Scalars* __restrict__ S) {
    pdl_entry_for(F, TMP, act, S);
    const int q = blockIdx.x;
    if (q >= n) return;
    const int tile = first + q;
    if (tile_done(tp, S, tile)) return;
    const int tt = meta_type(tp.meta[tile].packed);
    const size_t base = (size_t)tile * kTileCells;
    const bool has_child0 = child[(size_t)tile * 8] >= 0;
    for (int c = threadIdx.x; c < kTileCells; c += blockDim.x) {
        const int i = c >> 6, j = (c >> 3) & 7, k = c & 7;
        const uint8_t ct = act[base + c];
        const int ch = child[(size_t)tile * 8 + ((i >> 2) | ((j >> 2) << 1) | ((k >> 2) << 2))];
        auto child_sum = [&](uint8_t types) {
            float sum = 0.f;
            if (ch < 0) return sum;
            const size_t cb = (size_t)ch * kTileCells;
#pragma unroll
            for (int s = 0; s < 8; s++) {
                const int cid = cell_of(2 * (i & 3) + (s & 1), 2 * (j & 3) + ((s >> 1) & 1), 2 * (k & 3) + ((s >> 2) & 1));
                if (act[cb + cid] & types) sum = __fadd_rn(sum, TMP[cb + cid]);
            }
            return sum;
        };
        if (tt == NONLEAF_T) {
            if (!(ct & INTERIOR_C)) RHS[base + c] = 0.f;
            if (has_child0) RHS[base + c] = __fmul_rn(child_sum(INTERIOR_C), one_over_alpha);
        } else if (tt == LEAF_T) {
            if (ct & kTypedCell) RHS[base + c] = __fadd_rn(F[base + c], child_sum(kTypedCell));
        } else if (tt == GHOST_T) {
            if (ct & kTypedCell) RHS[base + c] = 0.f;
        }
    }
}

// ProlongateAndUpdate128 (src/GMGSolver.cu:345-380) with the AMG cell types, on every tile of
// the level: GHOST cells take the parent cell's x where INTERIOR, other tiles add prolong_coeff
// times it (fused); non-INTERIOR cells 0.
__global__ void __launch_bounds__(128) k_amg_prolong(Topo tp, int first, int n, float* X, const uint8_t* __restrict__ act, float pc,
                                                     const Scalars* __restrict__ S) {
    pdl_entry_for(act, S);
    const int q = blockIdx.x;
    if (q >= n) return;
    const int tile = first + q;
    if (tile_done(tp, S, tile)) return;
    const TileMeta m = tp.meta[tile];
    const bool ghost = meta_type(m.packed) & GHOST_T;
    const int oct = meta_octant(m.packed);
    const size_t base = (size_t)tile * kTileCells;
    for (int c = threadIdx.x; c < kTileCells; c += blockDim.x) {
        const int i = c >> 6, j = (c >> 3) & 7, k = c & 7;
        const float cx = m.parent < 0 ? 0.f
                                      : X[(size_t)m.parent * kTileCells +
                                          cell_of((oct & 1) * 4 + (i >> 1), ((oct >> 1) & 1) * 4 + (j >> 1), ((oct >> 2) & 1) * 4 + (k >> 1))];
        const bool interior = act[base + c] & INTERIOR_C;
        X[base + c] = !interior ? 0.f : ghost ? cx : fmaf(pc, cx, X[base + c]);
    }
}

// ---------------------------------------------------------------------------- fused V-cycle
// The V-cycle of the solves (level_iters 1) with four launches per level and one for level 0, the
// arithmetic of the kernels above operation by operation (the finite results are theirs bit for
// bit; only the sign of a zero right-hand side may differ, which no value of z depends on):
//   k_amg_presmooth       both colours of the downstroke's sweep from x = 0 into xpre: the first is
//                         pointwise, so the tile and its neighbours' first layer are formed in place
//   k_amg_residual_restrict  the residual and its 2x2x2 sums into the parent's right-hand side;
//                         GHOST tiles (x = 0, right-hand side 0) only where a face meets another tile
//   k_amg_level0          the coarsest level's sweeps, one CTA per instance
//   k_amg_prolong_sweep   prolongation of the tile and its halo, then the first colour
//   k_amg_sweep           the second colour, with the r.z part of its LEAF tiles
// What bounds them is memory latency and the coefficients' bytes: a cell's four planes are 16 of
// the 25 bytes a sweep reads.  Where a warp's 128 cells and the cells their upper faces take
// coefficients from all carry one off-diagonal and one diagonal (the fluid away from walls and
// level changes: most of a tree), k_amg_uniform notes the two numbers per warp and the planes are
// not read.  One tile per 128-thread CTA: the per-warp branch keeps the coefficients in registers,
// and the CTAs in flight, not the tiles per CTA, cover the latency.
// ring512 x4, the whole solve (30 iterations): 23.0 -> 10.5 ms; a level's four launches 13 us each
// over all levels, where the ten of the unfused V-cycle took 11-24 us.

// Per warp of a tile's 128-thread group (cells 128 w .. 128 w + 127): (off-diagonal, diagonal) where
// every cell is INTERIOR and has these on all faces, else (0, 0).
__global__ void __launch_bounds__(128) k_amg_uniform(Topo tp, int n, const uint8_t* __restrict__ act, const float* __restrict__ C,
                                                     size_t plane, float2* __restrict__ uni) {
    const int tile = blockIdx.x, t = threadIdx.x;
    if (tile >= n) return;
    const TileMeta m = tp.meta[tile];
    const TileIdx ix(t);
    const size_t base = (size_t)tile * kTileCells, o = base + t * 4;
    const uint32_t at = *reinterpret_cast<const uint32_t*>(act + o);
    const V4<float> cx = ld4(C + o), cy = ld4(C + plane + o), cz = ld4(C + 2 * plane + o), d = ld4(C + 3 * plane + o);
    const float c0 = __shfl_sync(0xffffffffu, cx.v[0], 0), d0 = __shfl_sync(0xffffffffu, d.v[0], 0);
    auto upper = [&](int axis, bool inside, int step) -> V4<float> {
        if (inside) return ld4(C + axis * plane + o + step);
        const int nb = m.nb[2 * axis + 1];
        return nb >= 0 ? ld4(C + axis * plane + (size_t)nb * kTileCells + (t * 4 - 7 * step)) : zero4<float>();
    };
    const V4<float> cxp = upper(0, ix.i < 7, 64), cyp = upper(1, ix.j < 7, 8);
    const float czp = ix.k0 == 0 ? C[2 * plane + o + 4] : m.nb[5] >= 0 ? C[2 * plane + (size_t)m.nb[5] * kTileCells + t * 4 - 4] : 0.f;
    bool same = at == 0x01010101u * INTERIOR_C && czp == c0 && d0 != 0.f;
#pragma unroll
    for (int e = 0; e < 4; e++)
        same = same && cx.v[e] == c0 && cy.v[e] == c0 && cz.v[e] == c0 && d.v[e] == d0 && cxp.v[e] == c0 && cyp.v[e] == c0;
    same = __all_sync(0xffffffffu, same);
    if ((t & 31) == 0) uni[(size_t)tile * 4 + (t >> 5)] = same ? make_float2(c0, d0) : make_float2(0.f, 0.f);
}

// The coefficients of thread t's column of four cells: the three lower faces, the upper x and y
// faces and the column's outer z+ face, the diagonal, and the AMG cell types.
struct AmgColumn {
    V4<float> cx, cy, cz, cxp, cyp, d;
    float czp;
    uint32_t ct;
};
__device__ __forceinline__ V4<float> splat4(float v) {
    V4<float> r;
    r.v[0] = r.v[1] = r.v[2] = r.v[3] = v;
    return r;
}
__device__ __forceinline__ void amg_column(AmgColumn& a, float2 u, const TileMeta& m, const float* __restrict__ C, size_t plane,
                                           const uint8_t* __restrict__ act, int tile, int t) {
    if (u.y != 0.f) {  // the whole warp
        a.cx = a.cy = a.cz = a.cxp = a.cyp = splat4(u.x);
        a.czp = u.x;
        a.d = splat4(u.y);
        a.ct = 0x01010101u * INTERIOR_C;
        return;
    }
    const TileIdx ix(t);
    const size_t o = (size_t)tile * kTileCells + t * 4;
    a.ct = *reinterpret_cast<const uint32_t*>(act + o);
    a.cx = ld4(C + o);
    a.cy = ld4(C + plane + o);
    a.cz = ld4(C + 2 * plane + o);
    a.d = ld4(C + 3 * plane + o);
    // an upper face's coefficient is the next cell's, 0 where that cell's tile is absent
    const int nx = ix.i < 7 ? tile : m.nb[1], ny = ix.j < 7 ? tile : m.nb[3], nz = ix.k0 == 0 ? tile : m.nb[5];
    a.cxp = nx >= 0 ? ld4(C + (size_t)nx * kTileCells + ((t * 4 + 64) & 511)) : zero4<float>();
    a.cyp = ny >= 0 ? ld4(C + plane + (size_t)ny * kTileCells + (ix.i * 64 + ((ix.j + 1) & 7) * 8 + ix.k0)) : zero4<float>();
    a.czp = nz >= 0 ? C[2 * plane + (size_t)nz * kTileCells + (ix.i * 64 + ix.j * 8 + (ix.k0 ^ 4))] : 0.f;
}
// amg_lap of cell e of the column, from its x and its neighbours'
__device__ __forceinline__ float column_lap(const AmgColumn& a, int e, float x0, float xm, float xp, float ym, float yp, float zl, float zr) {
    float s = __fmul_rn(x0, a.d.v[e]);
    s = fmaf(a.cx.v[e], xm, s);
    s = fmaf(a.cxp.v[e], xp, s);
    s = fmaf(a.cy.v[e], ym, s);
    s = fmaf(a.cyp.v[e], yp, s);
    s = fmaf(a.cz.v[e], zl, s);
    return fmaf(e < 3 ? a.cz.v[e < 3 ? e + 1 : 3] : a.czp, zr, s);
}
// The column's x and its neighbours' from a staged tile (xs, halos hx[6][64]).
struct AmgNeighbours {
    V4<float> xc, xm, xp, ym, yp;
    float zlo, zhi;
    __device__ __forceinline__ AmgNeighbours(const float* xs, const float* hx, int t) {
        const TileIdx ix(t);
        xc = ld4(xs + t * 4);
        xm = ld4(ix.i > 0 ? xs + (t - 16) * 4 : hx + 0 * 64 + ix.j * 8 + ix.k0);
        xp = ld4(ix.i < 7 ? xs + (t + 16) * 4 : hx + 1 * 64 + ix.j * 8 + ix.k0);
        ym = ld4(ix.j > 0 ? xs + (t - 2) * 4 : hx + 2 * 64 + ix.i * 8 + ix.k0);
        yp = ld4(ix.j < 7 ? xs + (t + 2) * 4 : hx + 3 * 64 + ix.i * 8 + ix.k0);
        zlo = *(ix.k0 > 0 ? xs + t * 4 - 1 : hx + 4 * 64 + ix.i * 8 + ix.j);
        zhi = *(ix.k0 < 4 ? xs + t * 4 + 4 : hx + 5 * 64 + ix.i * 8 + ix.j);
    }
    __device__ __forceinline__ float lap(const AmgColumn& a, int e) const {
        return column_lap(a, e, xc.v[e], xm.v[e], xp.v[e], ym.v[e], yp.v[e], e > 0 ? xc.v[e > 0 ? e - 1 : 0] : zlo,
                          e < 3 ? xc.v[e < 3 ? e + 1 : 3] : zhi);
    }
};
// One colour of the column: cells e = p and p + 2 with p = (color + i + j) & 1 (k0 is even).
__device__ __forceinline__ V4<float> amg_colour(const AmgColumn& a, const AmgNeighbours& x, const V4<float>& b, int t, int color) {
    const TileIdx ix(t);
    V4<float> o = x.xc;
    auto update = [&](int e) {
        float delta = 0.f;
        if ((a.ct >> (8 * e)) & INTERIOR_C) delta = __fdiv_rn(b.v[e] - x.lap(a, e), a.d.v[e]);
        o.v[e] = x.xc.v[e] + delta;
    };
    if ((color + ix.i + ix.j) & 1) {
        update(1);
        update(3);
    } else {
        update(0);
        update(2);
    }
    return o;
}
// a cell of the first colour from x = 0
__device__ __forceinline__ float amg_first(uint8_t ct, float b, float d) { return (ct & INTERIOR_C) ? 0.f + __fdiv_rn(b, d) : 0.f; }

// Offset of thread t's 4-cell piece of the x or y face f = t >> 4 (t < 64) in the neighbour's first
// layer, and of its cell of the z face 4 + (t >> 6): load_halo's pieces.
__device__ __forceinline__ int face_piece(int t) {
    const int f = t >> 4, q = t & 15;
    return f == 0 ? 448 + q * 4 : f == 1 ? q * 4 : f == 2 ? (q >> 1) * 64 + 56 + (q & 1) * 4 : (q >> 1) * 64 + (q & 1) * 4;
}
__device__ __forceinline__ int face_z_cell(int t) {
    const int c = t & 63;
    return (c >> 3) * 64 + (c & 7) * 8 + (t < 64 ? 7 : 0);
}

__global__ void __launch_bounds__(128) k_amg_presmooth(Topo tp, const int* __restrict__ list, float* __restrict__ XP,
                                                       const float* __restrict__ RHS, const uint8_t* __restrict__ act,
                                                       const float* __restrict__ C, size_t plane, const float2* __restrict__ uni,
                                                       const Scalars* __restrict__ S) {
    pdl_trigger();
    __shared__ __align__(16) TileShared<float> sh;
    const int t = threadIdx.x, tile = list[blockIdx.x];
    const TileMeta m = tp.meta[tile];
    const int fo = face_piece(t & 63), zo = face_z_cell(t), zf = 4 + (t >> 6);
    // GHOST neighbours hold x = 0 on the way down
    const int nf = t < 64 && !meta_nb_ghost(m.packed, t >> 4) ? m.nb[t >> 4] : -1, nz = meta_nb_ghost(m.packed, zf) ? -1 : m.nb[zf];
    pdl_wait_for(RHS, act, C, uni, S);
    if (tile_done(tp, S, tile)) return;
    const V4<float> b = ld4(RHS + (size_t)tile * kTileCells + t * 4);
    AmgColumn a;
    amg_column(a, uni[(size_t)tile * 4 + (t >> 5)], m, C, plane, act, tile, t);
    V4<float> hb = zero4<float>(), hd = splat4(1.f);
    uint32_t hct = 0;
    if (nf >= 0) {
        const size_t o = (size_t)nf * kTileCells + fo;
        hb = ld4(RHS + o);
        const float2 u = uni[(size_t)nf * 4 + (fo >> 7)];
        if (u.y != 0.f) {
            hd = splat4(u.y);
            hct = 0x01010101u * INTERIOR_C;
        } else {
            hd = ld4(C + 3 * plane + o);
            hct = *reinterpret_cast<const uint32_t*>(act + o);
        }
    }
    float zv = 0.f;
    if (nz >= 0 && (((zo >> 6) + (zo >> 3) + zo) & 1) == 0) {
        const size_t o = (size_t)nz * kTileCells + zo;
        zv = amg_first(act[o], RHS[o], C[3 * plane + o]);
    }
    const TileIdx ix(t);
    const int p = (ix.i + ix.j) & 1;
    V4<float> x = zero4<float>();
#pragma unroll
    for (int e = 0; e < 4; e++)
        if ((e & 1) == p) x.v[e] = amg_first((uint8_t)(a.ct >> (8 * e)), b.v[e], a.d.v[e]);
    st4(sh.xs + t * 4, x);
    if (t < 64) {
        const int hp = ((fo >> 6) + (fo >> 3)) & 1;  // the piece starts at an even k
        V4<float> h = zero4<float>();
#pragma unroll
        for (int e = 0; e < 4; e++)
            if ((e & 1) == hp) h.v[e] = amg_first((uint8_t)(hct >> (8 * e)), hb.v[e], hd.v[e]);
        st4(sh.hx + t * 4, h);
    }
    sh.hx[zf * 64 + (t & 63)] = zv;
    __syncthreads();
    st4(XP + (size_t)tile * kTileCells + t * 4, amg_colour(a, AmgNeighbours(sh.xs, sh.hx, t), b, t, 1));
}

// The residual of the 2x2x2 block c of a GHOST tile, summed as k_amg_restrict sums it, onto the
// LEAF parent's right-hand side.  x and the right-hand side are 0 on GHOST tiles, so only faces to
// other tiles contribute.
__device__ __forceinline__ void ghost_restrict(const Topo& tp, int tile, int c, const float* __restrict__ X, float* RHS,
                                               const uint8_t* __restrict__ act, const float* __restrict__ C, size_t plane) {
    const int fi = c / 16 * 2, fj = (c / 4) % 4 * 2, fk = c % 4 * 2;
    const TileMeta& m = tp.meta[tile];
    const uint32_t touch = (fi == 0 ? 1u : 0u) | (fi == 6 ? 2u : 0u) | (fj == 0 ? 4u : 0u) | (fj == 6 ? 8u : 0u) | (fk == 0 ? 16u : 0u) |
                           (fk == 6 ? 32u : 0u);
    uint32_t on = 0;
#pragma unroll
    for (int f = 0; f < 6; f++)
        if (((touch >> f) & 1u) && m.nb[f] >= 0 && !meta_nb_ghost(m.packed, f)) on |= 1u << f;
    if (on == 0 || m.parent < 0) return;
    const size_t base = (size_t)tile * kTileCells;
    float sum = 0.f;
#pragma unroll
    for (int s = 0; s < 8; s++) {  // x fastest
        const int ijk[3] = {fi + (s & 1), fj + ((s >> 1) & 1), fk + (s >> 2)};
        const int cell = cell_of(ijk[0], ijk[1], ijk[2]);
        float ax = 0.f;
        bool any = false;
#pragma unroll
        for (int f = 0; f < 6; f++) {
            const int axis = f >> 1, step = axis == 0 ? 64 : axis == 1 ? 8 : 1;
            if (!((on >> f) & 1u) || ijk[axis] != ((f & 1) ? 7 : 0)) continue;
            const size_t nb = (size_t)m.nb[f] * kTileCells + cell + ((f & 1) ? -7 * step : 7 * step);
            ax = fmaf(C[axis * plane + ((f & 1) ? nb : base + cell)], X[nb], ax);
            any = true;
        }
        if (any && act[base + cell] == INTERIOR_C) sum = __fadd_rn(sum, 0.f - ax);
    }
    const int oct = meta_octant(m.packed);
    float* out = RHS + (size_t)m.parent * kTileCells +
                 cell_of((oct & 1) * 4 + fi / 2, ((oct >> 1) & 1) * 4 + fj / 2, ((oct >> 2) & 1) * 4 + fk / 2);
    *out = __fadd_rn(*out, sum);
}
// The first ghost_blocks CTAs take the level's GHOST tiles, two each; the others list's tiles.
__global__ void __launch_bounds__(128) k_amg_residual_restrict(Topo tp, const int* __restrict__ list, const int* __restrict__ ghosts, int nghost,
                                                               int ghost_blocks, const float* __restrict__ X, float* RHS,
                                                               const uint8_t* __restrict__ act, const float* __restrict__ C, size_t plane,
                                                               const float2* __restrict__ uni, float one_over_alpha,
                                                               const Scalars* __restrict__ S) {
    pdl_trigger();
    const int t = threadIdx.x;
    if ((int)blockIdx.x < ghost_blocks) {
        const int q = (int)blockIdx.x * 2 + (t >> 6);
        const int tile = q < nghost ? ghosts[q] : -1;
        pdl_wait_for(X, RHS, act, C, S, uni);
        if (tile >= 0 && !tile_done(tp, S, tile)) ghost_restrict(tp, tile, t & 63, X, RHS, act, C, plane);
        return;
    }
    __shared__ __align__(16) TileShared<float> sh;
    const int tile = list[(int)blockIdx.x - ghost_blocks];
    const TileMeta m = tp.meta[tile];
    pdl_wait_for(X, RHS, act, C, uni, S);
    if (tile_done(tp, S, tile)) return;
    const V4<float> b = ld4(RHS + (size_t)tile * kTileCells + t * 4);
    AmgColumn a;
    amg_column(a, uni[(size_t)tile * 4 + (t >> 5)], m, C, plane, act, tile, t);
    stage_tile<float>(X, tile, m, t, sh);
    __syncthreads();
    const AmgNeighbours x(sh.xs, sh.hx, t);
    V4<float> r;
#pragma unroll
    for (int e = 0; e < 4; e++) r.v[e] = ((a.ct >> (8 * e)) & 0xffu) == INTERIOR_C ? b.v[e] - x.lap(a, e) : 0.f;
    __syncthreads();
    st4(sh.xs + t * 4, r);
    __syncthreads();
    if (t >= 64 || m.parent < 0) return;
    const int fi = t / 16 * 2, fj = (t / 4) % 4 * 2, fk = t % 4 * 2;
    float sum = 0.f;
#pragma unroll
    for (int s = 0; s < 8; s++) sum = __fadd_rn(sum, sh.xs[cell_of(fi + (s & 1), fj + ((s >> 1) & 1), fk + (s >> 2))]);
    const int oct = meta_octant(m.packed);
    RHS[(size_t)m.parent * kTileCells + cell_of((oct & 1) * 4 + fi / 2, ((oct >> 1) & 1) * 4 + fj / 2, ((oct >> 2) & 1) * 4 + fk / 2)] =
        __fmul_rn(sum, one_over_alpha);
}

// The level-0 sweeps of one instance (at most 8 tiles, coupled to no other instance's) in one CTA
// of 128 threads per tile: x in shared memory, every thread's coefficients and right-hand sides in
// registers, one barrier per colour.  Latency-bound: 20 sweeps of a two-tile level take 15 us
// (k_amg_gs_sequence, which re-reads x and the coefficients from memory each sweep: 40 us).
__global__ void __launch_bounds__(1024, 1) k_amg_level0(Topo tp, const int* __restrict__ list, const int2* __restrict__ ranges,
                                                        float* __restrict__ X, const float* __restrict__ RHS, const uint8_t* __restrict__ act,
                                                        const float* __restrict__ C, size_t plane, const float2* __restrict__ uni, int iters,
                                                        const Scalars* __restrict__ S) {
    pdl_trigger();
    __shared__ __align__(16) float xs[8][kTileCells];
    __shared__ __align__(16) float zero[64];
    __shared__ int tiles[8];
    const int2 r = ranges[blockIdx.x];
    const int g = threadIdx.x >> 7, t = threadIdx.x & 127;
    const bool on = g < r.y;
    const int tile = on ? list[r.x + g] : -1;
    if (t == 0) tiles[g] = tile;
    if (threadIdx.x < 64) zero[threadIdx.x] = 0.f;
    st4(&xs[g][t * 4], zero4<float>());
    TileMeta m;
    if (on) m = tp.meta[tile];
    __syncthreads();
    pdl_wait_for(RHS, act, C, uni, S);
    if (S && S[blockIdx.x].done) return;
    const TileIdx ix(t);
    // the column's neighbour vectors: in its own tile, in another of the instance's, or zeros
    const float *pxm = zero, *pxp = zero, *pym = zero, *pyp = zero, *pzl = zero, *pzr = zero;
    AmgColumn a;
    V4<float> b = zero4<float>();
    if (on) {
        auto where = [&](int f) {
            for (int k = 0; k < r.y; k++)
                if (tiles[k] == m.nb[f]) return k;
            return -1;  // absent, or GHOST (x = 0)
        };
        auto at = [&](bool inside, int f, int off) -> const float* {
            const int k = inside ? g : m.nb[f] >= 0 ? where(f) : -1;
            return k >= 0 ? &xs[k][off] : zero;
        };
        const int o = t * 4;
        pxm = at(ix.i > 0, 0, (o - 64) & 511);
        pxp = at(ix.i < 7, 1, (o + 64) & 511);
        pym = at(ix.j > 0, 2, ix.i * 64 + ((ix.j - 1) & 7) * 8 + ix.k0);
        pyp = at(ix.j < 7, 3, ix.i * 64 + ((ix.j + 1) & 7) * 8 + ix.k0);
        pzl = at(ix.k0 > 0, 4, ix.k0 > 0 ? o - 1 : o + 7);
        pzr = at(ix.k0 == 0, 5, ix.k0 == 0 ? o + 4 : o - 4);
        amg_column(a, uni[(size_t)tile * 4 + (t >> 5)], m, C, plane, act, tile, t);
        b = ld4(RHS + (size_t)tile * kTileCells + o);
    }
    const int q = (ix.i + ix.j) & 1;
    auto sweep = [&](int color) {
        if (on) {
            float* own = &xs[g][t * 4];
            const int p = (color + q) & 1;
            const V4<float> xc = ld4(own), xm = ld4(pxm), xp = ld4(pxp), ym = ld4(pym), yp = ld4(pyp);
            const float zl = *pzl, zr = *pzr;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if ((e & 1) != p) continue;
                float delta = 0.f;
                if ((a.ct >> (8 * e)) & INTERIOR_C) {
                    const float ax = column_lap(a, e, xc.v[e], xm.v[e], xp.v[e], ym.v[e], yp.v[e], e > 0 ? xc.v[e > 0 ? e - 1 : 0] : zl,
                                                e < 3 ? xc.v[e < 3 ? e + 1 : 3] : zr);
                    delta = __fdiv_rn(b.v[e] - ax, a.d.v[e]);
                }
                own[e] = xc.v[e] + delta;
            }
        }
        __syncthreads();
    };
    for (int it = 0; it < iters; it++) {
        sweep(0);
        sweep(1);
    }
    for (int it = 0; it < iters; it++) {
        sweep(1);
        sweep(0);
    }
    if (on) st4(X + (size_t)tile * kTileCells + t * 4, ld4(&xs[g][t * 4]));
}

// k_amg_prolong's value of a cell
__device__ __forceinline__ float amg_prolonged(uint8_t ct, bool ghost, float cx, float x, float pc) {
    return (ct & INTERIOR_C) ? (ghost ? cx : fmaf(pc, cx, x)) : 0.f;
}
// The first item_blocks CTAs prolongate the face layers of GHOST tiles that other tiles read, two
// items (tile, face, parent, octant) each; the others list's tiles: prolongation of the tile and its
// halo from the parents' Z and the pre-smoothed XP, then colour 1.
__global__ void __launch_bounds__(128) k_amg_prolong_sweep(Topo tp, const int* __restrict__ list, const int4* __restrict__ items, int nitems,
                                                           int item_blocks, float* Z, const float* __restrict__ XP,
                                                           const float* __restrict__ RHS, const uint8_t* __restrict__ act,
                                                           const float* __restrict__ C, size_t plane, const float2* __restrict__ uni, float pc,
                                                           const Scalars* __restrict__ S) {
    pdl_trigger();
    const int t = threadIdx.x;
    if ((int)blockIdx.x < item_blocks) {
        const int q = (int)blockIdx.x * 2 + (t >> 6);
        if (q >= nitems) {
            pdl_wait();
            return;
        }
        const int4 it = items[q];
        const int u = (t >> 3) & 7, v = t & 7;
        const int off = it.y < 2 ? (it.y & 1) * 448 + u * 8 + v : it.y < 4 ? u * 64 + (it.y & 1) * 56 + v : u * 64 + v * 8 + (it.y & 1) * 7;
        pdl_wait_for(Z, act, S, XP, RHS, C, uni);
        if (tile_done(tp, S, it.x)) return;
        const float cx = it.z >= 0 ? Z[(size_t)it.z * kTileCells + parent_cell(it.w, off)] : 0.f;
        const size_t o = (size_t)it.x * kTileCells + off;
        Z[o] = amg_prolonged(act[o], true, cx, 0.f, 0.f);
        return;
    }
    __shared__ __align__(16) TileShared<float> sh;
    const int tile = list[(int)blockIdx.x - item_blocks];
    const TileMeta m = tp.meta[tile];
    const TileIdx ix(t);
    const int fo = face_piece(t & 63), zo = face_z_cell(t), zf = 4 + (t >> 6);
    const int nf = t < 64 ? m.nb[t >> 4] : -1, nz = m.nb[zf];
    int fpar = -1, fpk = 0, zpar = -1, zpk = 0;
    if (nf >= 0) {
        fpar = tp.meta[nf].parent;
        fpk = tp.meta[nf].packed;
    }
    if (nz >= 0) {
        zpar = tp.meta[nz].parent;
        zpk = tp.meta[nz].packed;
    }
    const bool fghost = meta_type(fpk) & GHOST_T, zghost = meta_type(zpk) & GHOST_T;
    pdl_wait_for(Z, XP, RHS, act, C, uni, S);
    if (tile_done(tp, S, tile)) return;
    const size_t base = (size_t)tile * kTileCells;
    V4<float> x = ld4(XP + base + t * 4);
    const V4<float> b = ld4(RHS + base + t * 4);
    float2 c = make_float2(0.f, 0.f), hc = c;
    if (m.parent >= 0)
        c = *reinterpret_cast<const float2*>(Z + (size_t)m.parent * kTileCells + parent_cell(meta_octant(m.packed), t * 4));
    V4<float> h = zero4<float>();
    uint32_t hct = 0;
    if (nf >= 0) {
        const size_t o = (size_t)nf * kTileCells + fo;
        hct = *reinterpret_cast<const uint32_t*>(act + o);
        if (!fghost) h = ld4(XP + o);
        if (fpar >= 0) hc = *reinterpret_cast<const float2*>(Z + (size_t)fpar * kTileCells + parent_cell(meta_octant(fpk), fo));
    }
    float zv = 0.f;
    if (nz >= 0) {
        const size_t o = (size_t)nz * kTileCells + zo;
        const float zc = zpar >= 0 ? Z[(size_t)zpar * kTileCells + parent_cell(meta_octant(zpk), zo)] : 0.f;
        zv = amg_prolonged(act[o], zghost, zc, zghost ? 0.f : XP[o], pc);
    }
    AmgColumn a;
    amg_column(a, uni[(size_t)tile * 4 + (t >> 5)], m, C, plane, act, tile, t);
#pragma unroll
    for (int e = 0; e < 4; e++) x.v[e] = amg_prolonged((uint8_t)(a.ct >> (8 * e)), false, e < 2 ? c.x : c.y, x.v[e], pc);
    st4(sh.xs + t * 4, x);
    if (t < 64) {
#pragma unroll
        for (int e = 0; e < 4; e++) h.v[e] = amg_prolonged((uint8_t)(hct >> (8 * e)), fghost, e < 2 ? hc.x : hc.y, h.v[e], pc);
        st4(sh.hx + t * 4, h);
    }
    sh.hx[zf * 64 + (t & 63)] = zv;
    __syncthreads();
    st4(Z + base + t * 4, amg_colour(a, AmgNeighbours(sh.xs, sh.hx, t), b, t, 1));
}

// Colour 0 on list's tiles; with RD (the PCG residual) also the r.z part of the level's LEAF tiles
// at WP[LEAF slot], formed as the GMG V-cycle's last sweep forms it.
__global__ void __launch_bounds__(128) k_amg_sweep(Topo tp, const int* __restrict__ list, float* X, const float* __restrict__ RHS,
                                                   const uint8_t* __restrict__ act, const float* __restrict__ C, size_t plane,
                                                   const float2* __restrict__ uni, const Scalars* __restrict__ S, const float* __restrict__ RD,
                                                   double* __restrict__ WP) {
    pdl_trigger();
    __shared__ __align__(16) TileShared<float> sh;
    __shared__ __align__(16) float term[128];
    const int t = threadIdx.x, tile = list[blockIdx.x];
    const TileMeta m = tp.meta[tile];
    const int slot = tp.leafslot[tile];
    pdl_wait_for(X, RHS, act, C, uni, S, RD);
    if (tile_done(tp, S, tile)) return;
    const size_t o = (size_t)tile * kTileCells + t * 4;
    const V4<float> b = ld4(RHS + o);
    // the part's r: the right-hand side itself unless GHOST children added to it
    const V4<float> rd = RD != nullptr && slot < -1 ? ld4(RD + o) : b;
    AmgColumn a;
    amg_column(a, uni[(size_t)tile * 4 + (t >> 5)], m, C, plane, act, tile, t);
    stage_tile<float>(X, tile, m, t, sh);
    __syncthreads();
    const V4<float> z = amg_colour(a, AmgNeighbours(sh.xs, sh.hx, t), b, t, 0);
    st4(X + o, z);
    if (RD == nullptr || slot == -1) return;
    term[t] = dot4f32(rd, z);
    __syncthreads();
    if (t >= 32) return;
    const double d = tile_part_sum(term, t & 15);
    if (t == 0) WP[slot >= 0 ? slot : -2 - slot] = d;
}

size_t amg_plane(const DevGrid& g) { return (size_t)g.n * kTileCells; }

void amg_gauss_seidel(const DevGrid& g, int iters, int order, int level, float* X, const float* RHS, const Scalars* S, cudaStream_t s) {
    const int n = g.mg_count[level];
    if (n == 0) return;
    for (int it = 0; it < iters; it++)
        for (int color : {order, 1 - order}) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_gs, n, 128, 0, s, g.topo, g.d_mg + g.mg_offset[level], n, X, RHS, (const uint8_t*)g.d_amg_ct,
                                  (const float*)g.d_amg, amg_plane(g), color, S);
        }
}

}  // namespace

int amg_prepare(DevGrid& g, float one_over_alpha, cudaStream_t s) {
    const size_t cells = amg_plane(g);
    if (!g.d_amg) {
        if (device_malloc(&g.d_amg, 4 * cells * sizeof(float)) != cudaSuccess) return 3;
        if (device_malloc(&g.d_amg_ct, cells) != cudaSuccess) {
            cudaFree(g.d_amg);
            g.d_amg = nullptr;
            return 3;
        }
        if (device_malloc(&g.d_amg_uni, sizeof(float2) * 4 * (size_t)g.n) != cudaSuccess) {
            cudaFree(g.d_amg);
            cudaFree(g.d_amg_ct);
            g.d_amg = nullptr;
            g.d_amg_ct = nullptr;
            return 3;
        }
        g.bytes += 4 * cells * sizeof(float) + cells + sizeof(float2) * 4 * (size_t)g.n;
    }
    cudaMemsetAsync(g.d_amg, 0, 4 * cells * sizeof(float), s);
    k_amg_types<<<g.n, 128, 0, s>>>(g.topo, g.n, g.d_amg_ct);
    if (g.n_leafghost > 0) k_amg_coeffs<<<g.n_leafghost, 128, 0, s>>>(g.topo, g.d_leafghost, g.n_leafghost, g.d_amg_ct, g.d_amg, cells);
    for (int l = g.max_level; l >= 0; l--)
        if (g.level_count[l] > 0)
            k_amg_coarsen<<<g.level_count[l], 128, 0, s>>>(g.topo, g.d_child, g.level_first[l], g.level_count[l], g.d_amg_ct, g.d_amg, cells,
                                                           one_over_alpha);
    k_amg_uniform<<<g.n, 128, 0, s>>>(g.topo, g.n, g.d_amg_ct, g.d_amg, cells, g.d_amg_uni);
    g.launch_count += 3 + g.max_level + 1;
    if (cudaGetLastError() != cudaSuccess) return 2;
    // per instance, its entries of the level-0 LEAF|NONLEAF list (the list is instance by
    // instance): the coarsest level's sweeps run as one CTA per instance
    if (!g.d_amg_l0 && g.mg_count[0] > 0) {
        // from the host tables: the level-0 list holds the level's LEAF|NONLEAF tiles in pool
        // order, and each instance's tiles of a level are one run of the pool
        std::vector<int> inst(g.n, -1);
        for (int i = 0; i < g.num_inst; i++)
            for (const TileRun& r : g.inst_runs[i])
                for (int t = r.global; t < r.global + r.count; t++) inst[t] = i;
        std::vector<int2> ranges(g.num_inst, int2{0, 0});
        bool contiguous = true;
        int q = 0;
        for (int t = g.level_first[0]; t < g.level_first[0] + g.level_count[0]; t++) {
            if (!(g.h_tile_type[t] & (LEAF_T | NONLEAF_T))) continue;
            int2& r = ranges[inst[t]];
            if (r.y == 0) r.x = q;
            else if (r.x + r.y != q) contiguous = false;
            r.y++;
            q++;
        }
        if (q != g.mg_count[0]) contiguous = false;
        g.amg_l0_max = 0;
        if (contiguous)  // (else the sweeps take one launch each)
            for (const int2& r : ranges) g.amg_l0_max = std::max(g.amg_l0_max, (int)r.y);
        if (device_malloc(&g.d_amg_l0, sizeof(int2) * g.num_inst) != cudaSuccess) return 3;
        if (cudaMemcpy(g.d_amg_l0, ranges.data(), sizeof(int2) * g.num_inst, cudaMemcpyHostToDevice) != cudaSuccess) return 2;
    }
    g.amg_ready = true;
    return 0;
}

int amg_download(const DevGrid& g, float* coeffs, uint8_t* types, cudaStream_t s) {
    if (!g.amg_ready) return 1;
    const size_t cells = amg_plane(g);
    if (coeffs && cudaMemcpyAsync(coeffs, g.d_amg, 4 * cells * sizeof(float), cudaMemcpyDeviceToHost, s) != cudaSuccess) return 2;
    if (types && cudaMemcpyAsync(types, g.d_amg_ct, cells, cudaMemcpyDeviceToHost, s) != cudaSuccess) return 2;
    return cudaStreamSynchronize(s) == cudaSuccess ? 0 : 2;
}

// VCycleAMG (src/AMGSolver.cu:610-715): x = 0, rhs = f (0 on GHOST tiles); downstroke per level
// GaussSeidelAMG(level_iters, order 0), residual, restriction; level 0 GaussSeidelAMG(ci/2, 0) +
// GaussSeidelAMG(ci/2, 1); upstroke ProlongateAndUpdate128 + GaussSeidelAMG(level_iters, 1).
void vcycle_amg(const DevGrid& g, float* X, const float* F, float* TMP, float* RHS, int level_iters, int coarsest_iters,
                float one_over_alpha, float prolong_coeff, const Scalars* S, cudaStream_t s) {
    const size_t plane = amg_plane(g);
    launch::vcycle_init(g, X, RHS, F, S, s);
    for (int l = g.max_level; l > 0; l--) {
        amg_gauss_seidel(g, level_iters, 0, l, X, RHS, S, s);
        if (g.level_count[l] > 0) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_residual, g.level_count[l], 128, 0, s, g.topo, g.level_first[l], g.level_count[l], (const float*)X,
                                  (const float*)RHS, TMP, (const uint8_t*)g.d_amg_ct, (const float*)g.d_amg, plane, S);
        }
        if (g.level_count[l - 1] > 0) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_restrict, g.level_count[l - 1], 128, 0, s, g.topo, (const int*)g.d_child, g.level_first[l - 1],
                                  g.level_count[l - 1], F, (const float*)TMP, RHS, (const uint8_t*)g.d_amg_ct, one_over_alpha, S);
        }
    }
    // level 0: GaussSeidelAMG(ci/2, 0) + GaussSeidelAMG(ci/2, 1), as one sequence per instance
    // where every instance's level-0 tiles fit one CTA's rounds, else one launch per sweep
    if (g.d_amg_l0 && g.amg_l0_max > 0 && g.mg_count[0] > 0) {
        std::vector<int> cols;
        for (int it = 0; it < coarsest_iters / 2; it++) { cols.push_back(0); cols.push_back(1); }
        for (int it = 0; it < coarsest_iters / 2; it++) { cols.push_back(1); cols.push_back(0); }
        const int threads = 128 * std::min(8, g.amg_l0_max);
        for (size_t c0 = 0; c0 < cols.size(); c0 += 32) {
            uint32_t colors = 0;
            const int ns = (int)std::min<size_t>(32, cols.size() - c0);
            for (int k = 0; k < ns; k++) colors |= (uint32_t)cols[c0 + k] << k;
            ++g.launch_count;
            launch::launch_kernel(k_amg_gs_sequence, g.num_inst, threads, 0, s, g.topo, (const int*)(g.d_mg + g.mg_offset[0]),
                                  (const int2*)g.d_amg_l0, X, (const float*)RHS, (const uint8_t*)g.d_amg_ct, (const float*)g.d_amg, plane,
                                  colors, ns, S);
        }
    } else {
        amg_gauss_seidel(g, coarsest_iters / 2, 0, 0, X, RHS, S, s);
        amg_gauss_seidel(g, coarsest_iters / 2, 1, 0, X, RHS, S, s);
    }
    for (int l = 1; l <= g.max_level; l++) {
        if (g.level_count[l] > 0) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_prolong, g.level_count[l], 128, 0, s, g.topo, g.level_first[l], g.level_count[l], X,
                                  (const uint8_t*)g.d_amg_ct, prolong_coeff, S);
        }
        amg_gauss_seidel(g, level_iters, 1, l, X, RHS, S, s);
    }
}

// The fused V-cycle applies: one sweep per level, at most 8 level-0 tiles per instance, every
// non-GHOST tile under a NONLEAF one that has all eight children and every GHOST tile under a LEAF
// one (each right-hand side then has the one writer that the kernels give it).
bool amg_use_fused(const DevGrid& g, int level_iters) {
    const char* e = std::getenv("CIRRUS_VCYCLE");
    if (e && std::strcmp(e, "generic") == 0) return false;
    return level_iters == 1 && g.tree_regular && g.bottom_level >= 0 && g.d_amg_l0 && g.amg_l0_max > 0 && g.amg_l0_max <= 8;
}

void vcycle_amg_fused(const DevGrid& g, float* X, float* RHS, int coarsest_iters, float one_over_alpha, float prolong_coeff, const Scalars* S,
                      cudaStream_t s, const float* dot_r) {
    const size_t plane = amg_plane(g);
    const uint8_t* act = g.d_amg_ct;
    const float* C = g.d_amg;
    const float2* uni = g.d_amg_uni;
    float* XP = g.d_xpre;
    for (int l = g.max_level; l > 0; l--) {
        const int n = g.mg_count[l], ng = g.ghost_count[l], gb = (ng + 1) / 2;
        const int* list = g.d_mg + g.mg_offset[l];
        if (n > 0) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_presmooth, n, 128, 0, s, g.topo, list, XP, (const float*)RHS, act, C, plane, uni, S);
        }
        if (n + gb > 0) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_residual_restrict, gb + n, 128, 0, s, g.topo, list, g.d_ghost + g.ghost_offset[l], ng, gb,
                                  (const float*)XP, RHS, act, C, plane, uni, one_over_alpha, S);
        }
    }
    ++g.launch_count;
    launch::launch_kernel(k_amg_level0, g.num_inst, 128 * g.amg_l0_max, 0, s, g.topo, (const int*)(g.d_mg + g.mg_offset[0]),
                          (const int2*)g.d_amg_l0, X, (const float*)RHS, act, C, plane, uni, coarsest_iters / 2, S);
    for (int l = 1; l <= g.max_level; l++) {
        const int n = g.mg_count[l], ni = g.pri_cnt[l], ib = (ni + 1) / 2;
        const int* list = g.d_mg + g.mg_offset[l];
        if (n + ib > 0) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_prolong_sweep, ib + n, 128, 0, s, g.topo, list, (const int4*)(g.d_pritems + g.pri_off[l]), ni, ib, X,
                                  (const float*)XP, (const float*)RHS, act, C, plane, uni, prolong_coeff, S);
        }
        if (n > 0) {
            ++g.launch_count;
            launch::launch_kernel(k_amg_sweep, n, 128, 0, s, g.topo, list, X, (const float*)RHS, act, C, plane, uni, S, dot_r,
                                  dot_r ? g.d_wpart : (double*)nullptr);
        }
    }
    if (dot_r) launch::leaf_wpart(g, dot_r, X, s);
}

}  // namespace cirrus
