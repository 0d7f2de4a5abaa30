// Right-hand side of the pressure projection, built on the device as FluidEuler::project does
// (src/FluidEuler.h:583-586) after the velocity boundary step's face clearing
// (src/FluidEuler.cu:43-60).  Velocities live on the three lower faces of each cell
// (channels u, u+1, u+2); all arithmetic is FP32 as in the reference.
#include "kernels.cuh"
#include "solver_internal.hpp"

namespace cirrus {

namespace {

// Every kernel here takes one 128-thread group per tile, thread t owning the four cells 4t..4t+3 of
// a column, so that a channel is read and written in 16-byte vectors and a cell's neighbours inside
// the tile are other threads' vectors.  All are bound by bytes; what a tile does not need is not
// read (velocities of tiles without a face to clear, values inside GHOST tiles, whose cells only
// couple across faces to LEAF tiles).  ring512 x8 (40 k LEAF|GHOST tiles), us before (one cell at a
// time, one channel a launch) and now: face clearing 62, 28; propagation of the velocity 3 x 26, 30;
// divergence 144, 52 (4.2 TB/s of its DRAM bytes); its accumulation 43, 15; gradient 165, 107
// (3.8 TB/s); its accumulation 3 x 43, 13.

// ClearAllNeumannNeighborFaces on LEAF tiles: the lower face of axis a is zeroed when the cell
// or a cell across it is NEUMANN, or both are DIRICHLET.  Across a NONLEAF or GHOST neighbour
// the four finer cells behind the face are tested (IterateFaceNeighborCellTypes,
// src/PoissonGrid.h:451-489).
__device__ __forceinline__ bool clears(uint32_t t0, uint32_t t1) { return ((t0 | t1) & NEUMANN_C) || (t0 & t1 & DIRICHLET_C); }
// Most columns have nothing to clear, which their stencil masks (Laplacian context) tell in one
// load: an INTERIOR cell whose three lower faces carry coefficients has no NEUMANN cell across them.
// Only the others look at the types: 28 us for 20.7 k LEAF tiles, 43 with every column
// testing its types.  A mask knows the GHOST cell across a face but not the finer cells behind it, and
// an INTERIOR cell may be DIRICHLET as well, so every column tests where a GHOST tile has children or
// a cell is both (by_mask false).
__device__ __forceinline__ void clear_column(const Topo& tp, const int* __restrict__ child, int tile, int t, float* const (&U)[3]) {
    const TileMeta& m = tp.meta[tile];
    const TileIdx ix(t);
    const uint8_t* ct = tp.ctype + (size_t)tile * kTileCells + t * 4;
    const uint32_t own = *reinterpret_cast<const uint32_t*>(ct);
    // the types across the column's lower faces, tested where the tile across is LEAF (its own, for
    // the cells inside); the finer cells of another tile follow
    uint32_t across[3] = {0u, 0u, own << 8};
    bool tested[3];
    const int at[3] = {ix.i, ix.j, ix.k0};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int step = a == 0 ? 64 : a == 1 ? 8 : 1, nb = m.nb[2 * a];
        const uint8_t* nt = nullptr;
        if (at[a] > 0) nt = ct - step;
        else if (nb >= 0 && (meta_type(tp.meta[nb].packed) & LEAF_T)) nt = tp.ctype + (size_t)nb * kTileCells + t * 4 + 7 * step;
        tested[a] = nt != nullptr;
        if (nt == nullptr) continue;
        if (a < 2) across[a] = *reinterpret_cast<const uint32_t*>(nt);
        else across[a] |= *nt;
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        uint32_t set = 0u;
#pragma unroll
        for (int e = 0; e < 4; e++)
            if ((tested[a] || (a == 2 && e > 0)) && clears((own >> (8 * e)) & 0xffu, (across[a] >> (8 * e)) & 0xffu)) set |= 1u << e;
        const int nb = m.nb[2 * a];
        if (at[a] == 0 && !tested[a] && nb >= 0)
            for (int e = 0; e < (a == 2 ? 1 : 4); e++) {
                int nl[3] = {ix.i, ix.j, ix.k0 + e};
                nl[a] = 7;
                for (int q = 0; q < 4; q++) {
                    int off[3], c[3], oct = 0;
                    off[a] = 1;
                    off[(a + 1) % 3] = q >> 1;
                    off[(a + 2) % 3] = q & 1;
                    for (int d = 0; d < 3; d++) {
                        c[d] = nl[d] * 2 + off[d];
                        oct |= (c[d] >> 3) << d;
                    }
                    const int fine = child[(size_t)nb * 8 + oct];
                    if (fine >= 0 && clears((own >> (8 * e)) & 0xffu,
                                            tp.ctype[(size_t)fine * kTileCells + ((c[0] & 7) << 6 | (c[1] & 7) << 3 | (c[2] & 7))]))
                        set |= 1u << e;
                }
            }
        float* u = U[a] + (size_t)tile * kTileCells + t * 4;
        if (set == 15u) {
            st4(u, zero4<float>());
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if ((set >> e) & 1u) u[e] = 0.f;
        }
    }
}
__global__ void __launch_bounds__(128) k_clear_faces(Topo tp, const int* __restrict__ child, const int* __restrict__ list, bool by_mask,
                                                     float* U0, float* U1, float* U2) {
    pdl_trigger();
    constexpr uint32_t open = 0x01010101u * (1u | 4u | 16u | (uint32_t)kMaskInterior);
    const int tile = list[blockIdx.x], t = threadIdx.x;
    const uint32_t mask = *reinterpret_cast<const uint32_t*>(tp.mask_lap + (size_t)tile * kTileCells + t * 4);
    pdl_wait_for(U0, U1, U2);
    if (by_mask && (mask & open) == open) return;
    float* const U[3] = {U0, U1, U2};
    clear_column(tp, child, tile, t, U);
}

// PropagateToChildren(c, c, -1, GHOST, LAUNCH_SUBTREE, I|D|N) (src/PoissonGrid.cu:635-661) of N
// channels: typed GHOST cells copy their parent cell's value (0 if the parent cell is untyped or
// absent).
template <int N>
__global__ void __launch_bounds__(128) k_propagate_children(Topo tp, const int* __restrict__ list, float* X0, float* X1, float* X2) {
    pdl_trigger();
    const int tile = list[blockIdx.x], t = threadIdx.x;
    const TileMeta m = tp.meta[tile];
    const TileIdx ix(t);
    const size_t o = (size_t)tile * kTileCells + t * 4;
    const uint32_t ct = *reinterpret_cast<const uint32_t*>(tp.ctype + o);
    const int oct = meta_octant(m.packed);
    const size_t po = (size_t)(m.parent < 0 ? 0 : m.parent) * kTileCells + ((oct & 1) * 4 + (ix.i >> 1)) * 64 +
                      (((oct >> 1) & 1) * 4 + (ix.j >> 1)) * 8 + ((oct >> 2) & 1) * 4 + (ix.k0 >> 1);
    const uint32_t pt = m.parent < 0 ? 0u : *reinterpret_cast<const uint16_t*>(tp.ctype + po);
    pdl_wait_for(X0, X1, X2);
    float* X[3] = {X0, X1, X2};
#pragma unroll
    for (int a = 0; a < N; a++) {
        float2 v = make_float2(0.f, 0.f);
        if (m.parent >= 0) v = *reinterpret_cast<const float2*>(X[a] + po);
        if (!(pt & 7u)) v.x = 0.f;
        if (!((pt >> 8) & 7u)) v.y = 0.f;
        bool typed = true;
#pragma unroll
        for (int e = 0; e < 4; e++) typed = typed && ((ct >> (8 * e)) & 7u);
        if (typed) {
            V4<float> w;
            w.v[0] = w.v[1] = v.x;
            w.v[2] = w.v[3] = v.y;
            st4(X[a] + o, w);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if ((ct >> (8 * e)) & 7u) X[a][o + e] = e < 2 ? v.x : v.y;
        }
    }
}

// VelocityVolumeDivergenceOnLeafs (src/PoissonSolver.cu:66-137) on LEAF|GHOST tiles: the sum of
// outgoing face fluxes u*h*h over LEAF-LEAF, LEAF-GHOST and GHOST-LEAF faces on INTERIOR cells, the
// faces in (axis, -/+) order, u*h*h fused into the sum; across an absent tile the tile's own type
// and u = 0.
__global__ void __launch_bounds__(128, 16) k_divergence(Topo tp, const int* __restrict__ list, const float* __restrict__ U0,
                                                    const float* __restrict__ U1, const float* __restrict__ U2, float* __restrict__ B) {
    pdl_trigger();
    const int tile = list[blockIdx.x], t = threadIdx.x;
    const TileMeta m = tp.meta[tile];
    const TileIdx ix(t);
    const int tt = meta_type(m.packed);
    const float h = tile_level_const(tp, tile, meta_level(m.packed)).h;
    const size_t base = (size_t)tile * kTileCells, o = base + t * 4;
    const uint32_t ct = *reinterpret_cast<const uint32_t*>(tp.ctype + o);
    // a face carries a flux where its Laplacian coefficient class is not 0 (LEAF-LEAF, LEAF-GHOST
    // and GHOST-LEAF pairs, an absent tile counting as the own type): no neighbour's type is loaded
    const uint32_t cls = tp.fcls[tile];
    const bool inner = tt == LEAF_T;
    auto counts = [&](bool edge, int f) { return edge ? ((cls >> (2 * f)) & 3u) != 0u : inner; };
    const int nxp = ix.i == 7 ? m.nb[1] : tile, nyp = ix.j == 7 ? m.nb[3] : tile, nzp = ix.k0 == 4 ? m.nb[5] : tile;
    const bool xm = counts(ix.i == 0, 0), xp = counts(ix.i == 7, 1), ym = counts(ix.j == 0, 2), yp = counts(ix.j == 7, 3),
               zm = counts(ix.k0 == 0, 4), zp = counts(ix.k0 == 4, 5);
    pdl_wait_for(U0, U1, U2);
    const V4<float> z0 = zero4<float>();
    const V4<float> u0 = xm ? ld4(U0 + o) : z0;
    const V4<float> u1 = xp && nxp >= 0 ? ld4(U0 + (size_t)nxp * kTileCells + ((t * 4 + 64) & 511)) : z0;
    const V4<float> v0 = ym ? ld4(U1 + o) : z0;
    const V4<float> v1 = yp && nyp >= 0 ? ld4(U1 + (size_t)nyp * kTileCells + (ix.i * 64 + ((ix.j + 1) & 7) * 8 + ix.k0)) : z0;
    const V4<float> w0 = inner || zm ? ld4(U2 + o) : z0;
    const float w1 = zp && nzp >= 0 ? U2[(size_t)nzp * kTileCells + (ix.i * 64 + ix.j * 8 + (ix.k0 ^ 4))] : 0.f;
    V4<float> b;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        float sum = 0.f;
        auto add = [&](bool on, float u) {
            if (on) sum = fmaf(__fmul_rn(u, h), h, sum);
        };
        add(xm, -u0.v[e]);
        add(xp, u1.v[e]);
        add(ym, -v0.v[e]);
        add(yp, v1.v[e]);
        add(e > 0 ? inner : zm, -w0.v[e]);
        add(e < 3 ? inner : zp, e < 3 ? w0.v[e < 3 ? e + 1 : 3] : w1);
        b.v[e] = ((ct >> (8 * e)) & INTERIOR_C) ? sum : 0.f;
    }
    st4(B + o, b);
}

// AccumulateToParents (below) of the divergence (GRADIENT false, coefficient 1, INTERIOR cells of B0)
// or of the velocity update's three channels (1/4, INTERIOR|DIRICHLET) in a tree whose LEAF tiles have
// only GHOST children, one thread per coarse cell of each GHOST tile.  A GHOST cell's divergence is 0
// off the faces to LEAF tiles, its updated u off the lower ones, so only the coarse cells on such
// faces are summed, for u only the children in the face's layer.
template <bool GRADIENT>
__global__ void __launch_bounds__(128) k_accumulate_faces(Topo tp, const int* __restrict__ ghosts, int n, float* B0, float* B1, float* B2) {
    pdl_trigger();
    constexpr uint32_t kTypes = GRADIENT ? INTERIOR_C | DIRICHLET_C : INTERIOR_C;
    const int q = (int)blockIdx.x * 2 + ((int)threadIdx.x >> 6), c = threadIdx.x & 63;
    const int tile = ghosts[q < n ? q : 0];
    const uint32_t cls = tp.fcls[tile];
    const int ci = c >> 4, cj = (c >> 2) & 3, ck = c & 3;
    const int at[3] = {ci, cj, ck};
    uint32_t on = 0;  // faces to LEAF tiles that the coarse cell touches
#pragma unroll
    for (int f = 0; f < 6; f++)
        if (((cls >> (2 * f)) & 3u) && at[f >> 1] == ((f & 1) ? 3 : 0) && !(GRADIENT && (f & 1))) on |= 1u << f;
    const TileMeta& m = tp.meta[tile];
    const int oct = meta_octant(m.packed);
    const size_t base = (size_t)tile * kTileCells + 2 * ci * 64 + 2 * cj * 8 + 2 * ck;
    const size_t po = (size_t)(m.parent < 0 ? 0 : m.parent) * kTileCells + ((oct & 1) * 4 + ci) * 64 + (((oct >> 1) & 1) * 4 + cj) * 8 +
                      ((oct >> 2) & 1) * 4 + ck;
    if (q >= n || m.parent < 0 || !(tp.ctype[po] & kTypes)) on = 0;
    pdl_wait_for(B0, B1, B2);
    if (on == 0) return;
    uint32_t ok = 0;  // children of the types, x fastest
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const uint32_t pair = *reinterpret_cast<const uint16_t*>(tp.ctype + base + (s & 1) * 64 + (s >> 1) * 8);
        ok |= ((pair & kTypes) ? 1u : 0u) << s | (((pair >> 8) & kTypes) ? 1u : 0u) << (4 + s);
    }
    float* B[3] = {B0, B1, B2};
#pragma unroll
    for (int a = 0; a < (GRADIENT ? 3 : 1); a++) {
        if (GRADIENT && !((on >> (2 * a)) & 1u)) continue;
        float sum = 0.f;
#pragma unroll
        for (int s = 0; s < 8; s++) {
            const int d[3] = {s & 1, (s >> 1) & 1, s >> 2};
            if (GRADIENT && d[a] == 1) continue;
            if ((ok >> s) & 1u) sum += B[a][base + d[0] * 64 + d[1] * 8 + d[2]];
        }
        B[a][po] = fmaf(sum, GRADIENT ? 0.25f : 1.f, B[a][po]);
    }
}

// AccumulateToParents(b, b, -1, LEAF, LAUNCH_SUBTREE, cell_types, coeff, additive)
// (src/PoissonGrid.cu:721-755) of N channels: cells of LEAF tiles whose type is in cell_types add
// coeff times the sum of their children's values over children of those types (childCoord order, x
// fastest), for trees whose LEAF tiles may have other children.
template <int N>
__global__ void __launch_bounds__(128) k_accumulate_children(Topo tp, const int* __restrict__ child, const int* __restrict__ list, float* B0,
                                                             float* B1, float* B2, uint32_t cell_types, float coeff) {
    pdl_trigger();
    const int tile = list[blockIdx.x], t = threadIdx.x;
    const TileIdx ix(t);
    const size_t o = (size_t)tile * kTileCells + t * 4;
    const uint32_t ct = *reinterpret_cast<const uint32_t*>(tp.ctype + o);
    const int fine = child[(size_t)tile * 8 + ((ix.i >> 2) | ((ix.j >> 2) << 1) | ((ix.k0 >> 2) << 2))];
    pdl_wait_for(B0, B1, B2);
    if (fine < 0) return;
    // the column's children: rows (2i + a, 2j + b), eight cells along k
    const size_t fo = (size_t)fine * kTileCells + (2 * ix.i & 7) * 64 + (2 * ix.j & 7) * 8;
    uint2 ft[4];
#pragma unroll
    for (int q = 0; q < 4; q++) ft[q] = *reinterpret_cast<const uint2*>(tp.ctype + fo + (q & 1) * 64 + (q >> 1) * 8);
    float* B[3] = {B0, B1, B2};
#pragma unroll
    for (int a = 0; a < N; a++) {
        V4<float> lo[4], hi[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            lo[q] = ld4(B[a] + fo + (q & 1) * 64 + (q >> 1) * 8);
            hi[q] = ld4(B[a] + fo + (q & 1) * 64 + (q >> 1) * 8 + 4);
        }
        V4<float> b = ld4(B[a] + o);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int k = (2 * e + c) & 3;
                    const uint32_t type = ((e < 2 ? ft[q].x : ft[q].y) >> (8 * k)) & 0xffu;
                    if (type & cell_types) sum += e < 2 ? lo[q].v[k] : hi[q].v[k];
                }
            if ((ct >> (8 * e)) & cell_types) b.v[e] = fmaf(sum, coeff, b.v[e]);
        }
        st4(B[a] + o, b);
    }
}

// The face terms of AddGradientToFaceCenters (src/PoissonSolver.cu:144-200) on LEAF|GHOST tiles:
// on each lower face (x-, y-, z-) u += (p1 - p0) / dh with dh = h between LEAF cells and 1.5 h
// across a LEAF-GHOST face (no term otherwise, nor across a NEUMANN cell); p1, p0 the INTERIOR
// values (0 elsewhere); an absent neighbour counts as the cell's own tile and cell type with
// p0 = 0.  GHOST tiles start from u = 0.  Where h is a power of two the division by it is the
// multiplication by its exact reciprocal (the same real number, rounded once).
__global__ void __launch_bounds__(128, 12) k_gradient(Topo tp, const int* __restrict__ list, const float* __restrict__ P, float* U0, float* U1,
                                                  float* U2) {
    pdl_trigger();
    const int tile = list[blockIdx.x], t = threadIdx.x;
    const TileMeta m = tp.meta[tile];
    const TileIdx ix(t);
    const int tt = meta_type(m.packed);
    const bool ghost = tt == GHOST_T;
    const float h = tile_level_const(tp, tile, meta_level(m.packed)).h;
    const float h15 = (float)(1.5 * (double)h);
    const float rh = 1.f / h;
    const bool pow2 = (__float_as_uint(h) & 0x7fffffu) == 0u && (__float_as_uint(rh) & 0x7fffffu) == 0u && rh < 1e30f && rh > 1e-30f;
    const size_t o = (size_t)tile * kTileCells + t * 4;
    const uint32_t ct = *reinterpret_cast<const uint32_t*>(tp.ctype + o);
    const int at[3] = {ix.i, ix.j, ix.k0};
    // of the column's lower faces (the first cell's for z): 0 none, 1 h, 2 1.5 h, the Laplacian's
    // coefficient classes
    const uint32_t fcls = tp.fcls[tile];
    int cls[3];
    uint32_t nct[3];   // types across them
    size_t no[3];
    bool there[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int step = a == 0 ? 64 : a == 1 ? 8 : 1;
        const int nt = at[a] > 0 ? tile : m.nb[2 * a];
        cls[a] = at[a] > 0 ? (ghost ? 0 : 1) : (int)((fcls >> (4 * a)) & 3u);
        there[a] = nt >= 0;
        no[a] = (size_t)(nt < 0 ? tile : nt) * kTileCells + (at[a] > 0 ? t * 4 - step : t * 4 + 7 * step);
        nct[a] = ct;
        if (cls[a] && there[a]) nct[a] = a < 2 ? *reinterpret_cast<const uint32_t*>(tp.ctype + no[a]) : tp.ctype[no[a]];
    }
    if (there[2] || at[2] > 0) nct[2] = (ct << 8) | (nct[2] & 0xffu);
    else nct[2] = (ct << 8) | (ct & 0xffu);
    // cells that the accumulation adds to, if only 0: it leaves no -0 there
    const bool plus0 = tp.ghost_child[(size_t)tile * 8 + ((ix.i >> 2) | ((ix.j >> 2) << 1) | ((ix.k0 >> 2) << 2))] >= 0;
    pdl_wait_for(P, U0, U1, U2);
    const bool need = !ghost || cls[0] || cls[1] || cls[2];
    V4<float> p = zero4<float>(), q[3];
    if (need) p = ld4(P + o);
#pragma unroll
    for (int a = 0; a < 2; a++) q[a] = cls[a] && there[a] ? ld4(P + no[a]) : zero4<float>();
    q[2] = zero4<float>();
    if (cls[2] && there[2]) q[2].v[0] = P[no[2]];
#pragma unroll
    for (int e = 1; e < 4; e++) q[2].v[e] = p.v[e - 1];
    float* U[3] = {U0, U1, U2};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        V4<float> u = ghost ? zero4<float>() : ld4(U[a] + o);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint32_t c1 = (ct >> (8 * e)) & 0xffu, c0 = (nct[a] >> (8 * e)) & 0xffu;
            const int c = a == 2 && e > 0 ? (tt == LEAF_T ? 1 : 0) : cls[a];
            if (c != 0 && !((c1 | c0) & NEUMANN_C)) {
                // beyond an absent tile p0 = 0 (q is 0 there)
                const float p1 = (c1 & INTERIOR_C) ? p.v[e] : 0.f, p0 = (c0 & INTERIOR_C) ? q[a].v[e] : 0.f;
                const float g = c == 2 ? (p1 - p0) / h15 : pow2 ? __fmul_rn(p1 - p0, rh) : (p1 - p0) / h;
                u.v[e] = u.v[e] + g;
            }
            if (plus0 && (c1 & (INTERIOR_C | DIRICHLET_C))) u.v[e] = u.v[e] + 0.f;
        }
        st4(U[a] + o, u);
    }
}

}  // namespace

namespace launch {

void clear_neumann_faces(const DevGrid& g, int u_channel, cudaStream_t s) {
    if (g.n_leaf == 0) return;
    ++g.launch_count;
    launch_kernel(k_clear_faces, g.n_leaf, 128, 0, s, g.topo, (const int*)g.d_child, g.d_leaf, g.clear_by_mask, g.d_ch[u_channel],
                  g.d_ch[u_channel + 1], g.d_ch[u_channel + 2]);
}

void propagate_to_children(const DevGrid& g, int channel, cudaStream_t s) {
    if (g.n_ghost == 0) return;
    ++g.launch_count;
    launch_kernel(k_propagate_children<1>, g.n_ghost, 128, 0, s, g.topo, g.d_ghost, g.d_ch[channel], (float*)nullptr, (float*)nullptr);
}

namespace {
template <bool GRADIENT>
void accumulate_children(const DevGrid& g, float* B0, float* B1, float* B2, cudaStream_t s) {
    const int n = g.tree_regular ? g.n_ghost : g.n_leaf;
    if (n == 0) return;
    ++g.launch_count;
    if (g.tree_regular)
        launch_kernel(k_accumulate_faces<GRADIENT>, (n + 1) / 2, 128, 0, s, g.topo, g.d_ghost, n, B0, B1, B2);
    else
        launch_kernel(k_accumulate_children<GRADIENT ? 3 : 1>, n, 128, 0, s, g.topo, (const int*)g.d_child, g.d_leaf, B0, B1, B2,
                      (uint32_t)(GRADIENT ? INTERIOR_C | DIRICHLET_C : INTERIOR_C), GRADIENT ? 0.25f : 1.0f);
}
}  // namespace

void velocity_divergence(const DevGrid& g, int u_channel, int b_channel, cudaStream_t s) {
    if (g.n_leafghost == 0) return;
    ++g.launch_count;
    launch_kernel(k_divergence, g.n_leafghost, 128, 0, s, g.topo, g.d_leafghost, (const float*)g.d_ch[u_channel],
                  (const float*)g.d_ch[u_channel + 1], (const float*)g.d_ch[u_channel + 2], g.d_ch[b_channel]);
    accumulate_children<false>(g, g.d_ch[b_channel], nullptr, nullptr, s);
}

void projection_rhs(const DevGrid& g, int u_channel, int b_channel, cudaStream_t s) {
    clear_neumann_faces(g, u_channel, s);
    if (g.n_ghost > 0) {
        ++g.launch_count;
        launch_kernel(k_propagate_children<3>, g.n_ghost, 128, 0, s, g.topo, g.d_ghost, g.d_ch[u_channel], g.d_ch[u_channel + 1],
                      g.d_ch[u_channel + 2]);
    }
    velocity_divergence(g, u_channel, b_channel, s);
}

void add_gradient(const DevGrid& g, int p_channel, int u_channel, cudaStream_t s) {
    propagate_ghosts<float>(g, g.d_ch[p_channel], nullptr, s);
    float *U0 = g.d_ch[u_channel], *U1 = g.d_ch[u_channel + 1], *U2 = g.d_ch[u_channel + 2];
    if (g.n_leafghost > 0) {
        ++g.launch_count;
        launch_kernel(k_gradient, g.n_leafghost, 128, 0, s, g.topo, g.d_leafghost, (const float*)g.d_ch[p_channel], U0, U1, U2);
    }
    accumulate_children<true>(g, U0, U1, U2, s);
}

}  // namespace launch
}  // namespace cirrus
