// The V-cycle's level kernels with 256 threads per tile and one tile per CTA (launch shape 6): for
// levels of few tiles, where a launch is as long as one warp's instruction stream -- a 128-thread
// group issues some 740 instructions per warp for a pre-smoothed tile -- and not bound by what the
// SMs issue together.  Thread t owns the pair of cells (i, j, k0), (i, j, k0 + 1), one of either
// colour, so a colour sweep is one cell, one division, per thread; the 192 halo pairs (6 faces of 32)
// go to the first 192 threads.  The arithmetic is that of the 128-thread kernels cell by cell, and
// so are the bits.  A chain of the same launch on ring512, us per launch with 128 threads and with
// 256, levels 3, 4, 5, 6 (192, 384, 768, 1472 tiles): pre-smoother 3.8 4.7 5.0 5.1, 3.3 3.1 3.7 6.0;
// residual 3.8 4.1 4.3 4.8, 3.1 3.4 3.4 4.9; prolongation 3.2 4.0 4.4 5.3, 1.9 3.1 3.2 5.6; last
// sweep 3.1 3.9 4.0 4.2, 3.1 2.9 3.8 4.9.
#include "kernels.cuh"
#include "solver_internal.hpp"

namespace cirrus {

namespace {

struct PairIdx {
    int i, j, k0;
    __device__ __forceinline__ explicit PairIdx(int t) : i(t >> 5), j((t >> 2) & 7), k0((t & 3) << 1) {}
};

// Pair u (0..31) of face f's halo: slots h, h + 1 of hx[f][64] and the offsets of their cells in the
// neighbour's first layer (x and y faces: [j or i][k], along k; z faces: [i][j], along j).
struct HaloPair {
    int h, off, step;
    __device__ __forceinline__ HaloPair(int f, int u) {
        const int a = u >> 2, b = (u & 3) << 1;
        h = a * 8 + b;
        step = f < 4 ? 1 : 8;
        off = f < 2 ? (f == 0 ? 448 : 0) + a * 8 + b : f < 4 ? a * 64 + (f == 2 ? 56 : 0) + b : a * 64 + b * 8 + (f == 4 ? 7 : 0);
    }
};

struct __align__(16) WideStage {
    float xs[kTileCells];
    float hx[6 * 64];
};

__device__ __forceinline__ float cross_coef(uint32_t cls, int f, const LevelConst<float>& L) { return ((cls >> (2 * f)) & 3u) == 2u ? L.c2 : L.c1; }

// The first colour (x = b/D from x = 0) of one cell; uniform warps by vote, as first_colour_run.
__device__ __forceinline__ float first_cell(int i, int j, int k, uint32_t m, float b, uint32_t cls, const LevelConst<float>& L) {
    float d;
    if (__all_sync(__activemask(), m == (uint32_t)kMaskFull)) {
        d = L.dfast;
    } else {
        const FaceCoef<float> C = face_coef(i, j, k, cls, L);  // (its z entries are for 4-cell runs: not used)
        d = diag_cell(m, C, k == 0 ? cross_coef(cls, 4, L) : L.c1, k == 7 ? cross_coef(cls, 5, L) : L.c1, L);
    }
    return (m & kMaskInterior) ? 0.f + (b - 0.f) / d : 0.f;
}

// The update of cell (i, j, k) of a staged tile with mask byte m and right-hand side b.
__device__ __forceinline__ float sweep_cell(const WideStage& st, int i, int j, int k, uint32_t m, float b, uint32_t cls, const LevelConst<float>& L) {
    const int c = i * 64 + j * 8 + k;
    const float x0 = st.xs[c];
    const float xm = i > 0 ? st.xs[c - 64] : st.hx[j * 8 + k];
    const float xp = i < 7 ? st.xs[c + 64] : st.hx[64 + j * 8 + k];
    const float ym = j > 0 ? st.xs[c - 8] : st.hx[128 + i * 8 + k];
    const float yp = j < 7 ? st.xs[c + 8] : st.hx[192 + i * 8 + k];
    const float zl = k > 0 ? st.xs[c - 1] : st.hx[256 + i * 8 + j];
    const float zr = k < 7 ? st.xs[c + 1] : st.hx[320 + i * 8 + j];
    if (__all_sync(__activemask(), m == (uint32_t)kMaskFull)) return gs_cell_fast(x0, xm, xp, ym, yp, zl, zr, b, L);
    const FaceCoef<float> C = face_coef(i, j, k, cls, L);
    return gs_cell(x0, xm, xp, ym, yp, zl, zr, b, m, C, k == 0 ? cross_coef(cls, 4, L) : L.c1, k == 7 ? cross_coef(cls, 5, L) : L.c1, L);
}

// Copies the tile and its face halos of channel X: 128 threads the tile's 16-byte vectors and a z
// face cell each, 64 more the x and y faces (nb: the neighbour of the thread's piece).
__device__ __forceinline__ int stage_face(int t) { return t < 128 ? 4 + (t >> 6) : t < 192 ? (t - 128) >> 4 : -1; }
__device__ __forceinline__ void stage_wide(const float* X, int tile, int nb, int t, WideStage& st) {
    if (t < 128) {
        cp_async16(st.xs + t * 4, X + (size_t)tile * kTileCells + t * 4);
        const int c = t & 63;
        float* d = st.hx + (4 + (t >> 6)) * 64 + c;
        if (nb >= 0) cp_async4(d, X + (size_t)nb * kTileCells + (c >> 3) * 64 + (c & 7) * 8 + (t < 64 ? 7 : 0));
        else *d = 0.f;
    } else if (t < 192) {
        const int f = (t - 128) >> 4, q = t & 15;
        const int off = f == 0 ? 448 + q * 4 : f == 1 ? q * 4 : f == 2 ? (q >> 1) * 64 + 56 + (q & 1) * 4 : (q >> 1) * 64 + (q & 1) * 4;
        float* d = st.hx + f * 64 + q * 4;
        if (nb >= 0) cp_async16(d, X + (size_t)nb * kTileCells + off);
        else st4(d, zero4<float>());
    }
}

// k_presmooth (vcycle_fused.cu)
__global__ void __launch_bounds__(256) k_presmooth_wide(Topo tp, const int* __restrict__ list, float* XP, const float* RHS, const Scalars* S) {
    pdl_trigger();
    __shared__ WideStage st;
    const int t = threadIdx.x, tile = list[blockIdx.x];
    const PairIdx ix(t);
    const TileMeta& m = tp.meta[tile];
    const int packed = m.packed, f = t >> 5;
    const uint32_t cls = tp.fcls[tile] >> 12;
    const size_t o = (size_t)tile * kTileCells + t * 2;
    const uint32_t mk = *reinterpret_cast<const uint16_t*>(tp.mask_mg + o);
    const LevelConst<float> L = tile_level_const(tp, tile, meta_level(packed));
    const HaloPair hp(f < 6 ? f : 0, t & 31);
    // the halo pair's colour-0 cell; GHOST neighbours hold x = 0
    const int hq = ((hp.off >> 6) + (hp.off >> 3) + hp.off) & 1, hc = hp.off + hq * hp.step;
    const int nb = f < 6 && !meta_nb_ghost(packed, f) ? m.nb[f] : -1;
    uint32_t hm = 0, hcls = 0;
    if (nb >= 0) {
        hm = tp.mask_mg[(size_t)nb * kTileCells + hc];
        hcls = tp.fcls[nb] >> 12;
    }
    pdl_wait_for(XP, RHS, S);
    const float2 b = *reinterpret_cast<const float2*>(RHS + o);
    const float hb = nb >= 0 ? RHS[(size_t)nb * kTileCells + hc] : 0.f;
    if (tile_done(tp, S, tile)) return;
    const int p = (ix.i + ix.j) & 1;  // the pair's colour-0 cell
    const float v = first_cell(ix.i, ix.j, ix.k0 + p, (mk >> (8 * p)) & 0xffu, p ? b.y : b.x, cls, L);
    *reinterpret_cast<float2*>(st.xs + t * 2) = p ? make_float2(0.f, v) : make_float2(v, 0.f);
    if (f < 6) {
        float h = 0.f;
        if (nb >= 0) h = first_cell(hc >> 6, (hc >> 3) & 7, hc & 7, hm, hb, hcls, L);
        *reinterpret_cast<float2*>(st.hx + f * 64 + hp.h) = hq ? make_float2(0.f, h) : make_float2(h, 0.f);
    }
    __syncthreads();
    const int e = 1 - p;
    const float w = sweep_cell(st, ix.i, ix.j, ix.k0 + e, (mk >> (8 * e)) & 0xffu, e ? b.y : b.x, cls, L);
    *reinterpret_cast<float2*>(XP + o) = e ? make_float2(v, w) : make_float2(w, v);
}

// k_gs_sweep, with the r.z parts of the level's LEAF tiles where RD is given
__global__ void __launch_bounds__(256) k_gs_sweep_wide(Topo tp, const int* __restrict__ list, float* X, const float* R, int color,
                                                       const Scalars* S, const float* RD, double* WP) {
    pdl_trigger();
    __shared__ WideStage st;
    __shared__ __align__(16) float term[128];
    const int t = threadIdx.x, tile = list[blockIdx.x], f = stage_face(t);
    const PairIdx ix(t);
    const TileMeta& m = tp.meta[tile];
    const int nb = f >= 0 ? m.nb[f] : -1;
    const uint32_t cls = tp.fcls[tile] >> 12;
    const size_t o = (size_t)tile * kTileCells + t * 2;
    const uint32_t mk = *reinterpret_cast<const uint16_t*>(tp.mask_mg + o);
    const LevelConst<float> L = tile_level_const(tp, tile, meta_level(m.packed));
    const int slot = RD != nullptr ? tp.leafslot[tile] : -1;
    pdl_wait_for(X, R, S, RD, WP);
    stage_wide(X, tile, nb, t, st);
    const float2 b = *reinterpret_cast<const float2*>(R + o);
    // the part's r: the right-hand side itself unless GHOST children added to it
    float2 rd = b;
    if (slot < -1) rd = *reinterpret_cast<const float2*>(RD + o);
    const bool done = tile_done(tp, S, tile);
    cp_async_wait_all();
    if (done) return;
    __syncthreads();
    const int e = (color + ix.i + ix.j) & 1;
    const float w = sweep_cell(st, ix.i, ix.j, ix.k0 + e, (mk >> (8 * e)) & 0xffu, e ? b.y : b.x, cls, L);
    float2 z = *reinterpret_cast<const float2*>(st.xs + t * 2);
    if (e) z.y = w;
    else z.x = w;
    *reinterpret_cast<float2*>(X + o) = z;
    if (slot == -1) return;
    // dot4f32 of the 4-cell vector held by two threads
    const float lo = fmaf(rd.x, z.x, rd.y * z.y);
    const float from = __shfl_up_sync(0xffffffffu, lo, 1);
    if (t & 1) term[t >> 1] = fmaf(rd.y, z.y, fmaf(rd.x, z.x, from));
    __syncthreads();
    if (t >= 32) return;
    const double d = tile_part_sum(term, t & 15);
    if (t == 0) WP[slot >= 0 ? slot : -2 - slot] = d;
}

// k_residual_restrict's staged path; ghost: a GHOST tile's sums are added
__global__ void __launch_bounds__(256) k_residual_wide(Topo tp, const int* __restrict__ list, const int4* __restrict__ items, int nitems,
                                                       int item_blocks, const float* X, const float* RHS, float* C, float one_over_alpha,
                                                       const Scalars* S) {
    pdl_trigger();
    const int t = threadIdx.x;
    if ((int)blockIdx.x < item_blocks) {
        const int q = (int)blockIdx.x * 256 + t;
        const int4 it = items[q < nitems ? q : 0];
        pdl_wait_for(X, C, S);
        if (q < nitems && !(S != nullptr && S[it.w / kLevelSlots].done)) ghost_face_restrict(tp, X, it, C);
        return;
    }
    __shared__ WideStage st;
    __shared__ __align__(16) float res[kTileCells];
    const int tile = list[(int)blockIdx.x - item_blocks], f = stage_face(t);
    const PairIdx ix(t);
    const TileMeta& m = tp.meta[tile];
    const int nb = f >= 0 ? m.nb[f] : -1, parent = m.parent, packed = m.packed;
    const uint32_t cls = tp.fcls[tile] >> 12;
    const size_t o = (size_t)tile * kTileCells + t * 2;
    const uint32_t mk = *reinterpret_cast<const uint16_t*>(tp.mask_mg + o);
    const LevelConst<float> L = tile_level_const(tp, tile, meta_level(packed));
    pdl_wait_for(X, RHS, C, S);
    stage_wide(X, tile, nb, t, st);
    const float2 b = *reinterpret_cast<const float2*>(RHS + o);
    const bool done = tile_done(tp, S, tile);
    cp_async_wait_all();
    if (done) return;
    __syncthreads();
    const int c = t * 2, jk = ix.j * 8 + ix.k0, ik = ix.i * 8 + ix.k0, ij = ix.i * 8 + ix.j;
    auto ld2 = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
    const float2 xc = ld2(st.xs + c);
    const float2 xm = ld2(ix.i > 0 ? st.xs + c - 64 : st.hx + jk), xp = ld2(ix.i < 7 ? st.xs + c + 64 : st.hx + 64 + jk);
    const float2 ym = ld2(ix.j > 0 ? st.xs + c - 8 : st.hx + 128 + ik), yp = ld2(ix.j < 7 ? st.xs + c + 8 : st.hx + 192 + ik);
    const float zl = *(ix.k0 > 0 ? st.xs + c - 1 : st.hx + 256 + ij), zr = *(ix.k0 < 6 ? st.xs + c + 2 : st.hx + 320 + ij);
    float a0, a1;  // A x
    if (__all_sync(0xffffffffu, mk == 0x7F7Fu)) {
        auto lap = [&](float x0, float m0, float m1, float m2, float m3, float m4, float m5) {
            float s = 0.f;
            s = fmaf(L.c1, x0 - m0, s);
            s = fmaf(L.c1, x0 - m1, s);
            s = fmaf(L.c1, x0 - m2, s);
            s = fmaf(L.c1, x0 - m3, s);
            s = fmaf(L.c1, x0 - m4, s);
            s = fmaf(L.c1, x0 - m5, s);
            return mul_h3(s, L.h);
        };
        a0 = lap(xc.x, xm.x, xp.x, ym.x, yp.x, zl, xc.y);
        a1 = lap(xc.y, xm.y, xp.y, ym.y, yp.y, xc.x, zr);
    } else {
        const float cxm = ix.i == 0 ? cross_coef(cls, 0, L) : L.c1, cxp = ix.i == 7 ? cross_coef(cls, 1, L) : L.c1;
        const float cym = ix.j == 0 ? cross_coef(cls, 2, L) : L.c1, cyp = ix.j == 7 ? cross_coef(cls, 3, L) : L.c1;
        const float czm = ix.k0 == 0 ? cross_coef(cls, 4, L) : L.c1, czp = ix.k0 == 6 ? cross_coef(cls, 5, L) : L.c1;
        auto lap = [&](uint32_t mm, float zm, float zp, float x0, float m0, float m1, float m2, float m3, float m4, float m5) {
            float s = 0.f;
            s = fmaf((mm & 1u) ? cxm : 0.f, x0 - m0, s);
            s = fmaf((mm & 2u) ? cxp : 0.f, x0 - m1, s);
            s = fmaf((mm & 4u) ? cym : 0.f, x0 - m2, s);
            s = fmaf((mm & 8u) ? cyp : 0.f, x0 - m3, s);
            s = fmaf((mm & 16u) ? zm : 0.f, x0 - m4, s);
            s = fmaf((mm & 32u) ? zp : 0.f, x0 - m5, s);
            return (mm & kMaskInterior) ? mul_h3(s, L.h) : 0.f;
        };
        a0 = lap(mk & 0xffu, czm, L.c1, xc.x, xm.x, xp.x, ym.x, yp.x, zl, xc.y);
        a1 = lap(mk >> 8, L.c1, czp, xc.y, xm.y, xp.y, ym.y, yp.y, xc.x, zr);
    }
    *reinterpret_cast<float2*>(res + c) = make_float2(b.x - a0, b.y - a1);
    __syncthreads();
    if (t >= 64 || parent < 0) return;
    const int fi = t / 16 * 2, fj = (t / 4) % 4 * 2, fk = t % 4 * 2;
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) sum += res[(fi + (q >> 2)) * 64 + (fj + ((q >> 1) & 1)) * 8 + fk + (q & 1)];
    const int oct = meta_octant(packed);
    const size_t pid = (size_t)parent * kTileCells + ((oct & 1) * 4 + fi / 2) * 64 + (((oct >> 1) & 1) * 4 + fj / 2) * 8 + ((oct >> 2) & 1) * 4 + fk / 2;
    if (meta_type(packed) & GHOST_T) C[pid] += sum;
    else C[pid] = sum * one_over_alpha;
}

// k_prolong_sweep; the first item_blocks CTAs prolongate GHOST face layers, four items each
__global__ void __launch_bounds__(256) k_prolong_wide(Topo tp, const int* __restrict__ list, const int4* __restrict__ items, int nitems,
                                                      int item_blocks, float* Z, const float* XP, const float* RHS, float prolong_coeff,
                                                      const Scalars* S) {
    pdl_trigger();
    const int t = threadIdx.x;
    if ((int)blockIdx.x < item_blocks) {
        const int q = (int)blockIdx.x * 4 + (t >> 6);
        const int4 it = items[q < nitems ? q : 0];
        pdl_wait_for(Z, S);
        if (q < nitems && !tile_done(tp, S, it.x)) ghost_face_prolong(tp, Z, it, t & 63);
        return;
    }
    __shared__ WideStage st;
    const int tile = list[(int)blockIdx.x - item_blocks], f = t >> 5;
    const PairIdx ix(t);
    const TileMeta& m = tp.meta[tile];
    const int packed = m.packed, parent = m.parent, nb = f < 6 ? m.nb[f] : -1;
    const uint32_t cls = tp.fcls[tile] >> 12;
    const size_t o = (size_t)tile * kTileCells + t * 2;
    const uint32_t mk = *reinterpret_cast<const uint16_t*>(tp.mask_mg + o);
    const LevelConst<float> L = tile_level_const(tp, tile, meta_level(packed));
    const HaloPair hp(f < 6 ? f : 0, t & 31);
    uint32_t hm0 = 0, hm1 = 0;
    int npar = -1, npk = 0;
    size_t no = 0;
    if (nb >= 0) {
        no = (size_t)nb * kTileCells + hp.off;
        hm0 = tp.mask_mg[no];
        hm1 = tp.mask_mg[no + hp.step];
        npar = tp.meta[nb].parent;
        npk = tp.meta[nb].packed;
    }
    const bool nghost = meta_type(npk) & GHOST_T;
    pdl_wait_for(Z, XP, RHS, S);
    const float2 x = *reinterpret_cast<const float2*>(XP + o), b = *reinterpret_cast<const float2*>(RHS + o);
    // a pair lies over one coarse cell
    const float cx = parent >= 0 ? Z[(size_t)parent * kTileCells + parent_cell(meta_octant(packed), t * 2)] : 0.f;
    float h0 = 0.f, h1 = 0.f, hcx = 0.f;
    if (nb >= 0) {
        if (!nghost) {
            h0 = XP[no];
            h1 = XP[no + hp.step];
        }
        if (npar >= 0) hcx = Z[(size_t)npar * kTileCells + parent_cell(meta_octant(npk), hp.off)];
    }
    if (tile_done(tp, S, tile)) return;
    float2 z = make_float2(prolong_value(mk & 0xffu, false, cx, x.x, prolong_coeff), prolong_value(mk >> 8, false, cx, x.y, prolong_coeff));
    *reinterpret_cast<float2*>(st.xs + t * 2) = z;
    if (f < 6)
        *reinterpret_cast<float2*>(st.hx + f * 64 + hp.h) = make_float2(
            nb >= 0 ? prolong_value(hm0, nghost, hcx, h0, prolong_coeff) : 0.f, nb >= 0 ? prolong_value(hm1, nghost, hcx, h1, prolong_coeff) : 0.f);
    __syncthreads();
    const int e = (1 + ix.i + ix.j) & 1;
    const float w = sweep_cell(st, ix.i, ix.j, ix.k0 + e, (mk >> (8 * e)) & 0xffu, e ? b.y : b.x, cls, L);
    if (e) z.y = w;
    else z.x = w;
    *reinterpret_cast<float2*>(Z + o) = z;
}

}  // namespace

namespace launch {

void presmooth_wide(const DevGrid& g, int level, float* XP, const float* RHS, const Scalars* S, cudaStream_t s) {
    launch_kernel(k_presmooth_wide, g.mg_count[level], 256, 0, s, g.topo, g.d_mg + g.mg_offset[level], XP, RHS, S);
}
void gs_sweep_wide(const DevGrid& g, int level, float* X, const float* R, int color, const Scalars* S, cudaStream_t s, const float* RD) {
    launch_kernel(k_gs_sweep_wide, g.mg_count[level], 256, 0, s, g.topo, g.d_mg + g.mg_offset[level], X, R, color, S, RD, g.d_wpart);
}
void residual_wide(const DevGrid& g, int level, const float* X, const float* RHS, float* C, float one_over_alpha, const Scalars* S, cudaStream_t s) {
    const int ni = g.rri_cnt[level], ib = (ni + 255) / 256;
    if (ib + g.rr_cnt[level] == 0) return;
    launch_kernel(k_residual_wide, ib + g.rr_cnt[level], 256, 0, s, g.topo, (const int*)(g.d_rrmain + g.rr_off[level]),
                  (const int4*)(g.d_rritems + g.rri_off[level]), ni, ib, X, RHS, C, one_over_alpha, S);
}
void prolong_wide(const DevGrid& g, int level, float* Z, const float* XP, const float* RHS, float prolong_coeff, const Scalars* S, cudaStream_t s) {
    const int ni = g.pri_cnt[level], ib = (ni + 3) / 4;
    if (ib + g.pr_cnt[level] == 0) return;
    launch_kernel(k_prolong_wide, ib + g.pr_cnt[level], 256, 0, s, g.topo, (const int*)(g.d_prmain + g.pr_off[level]),
                  (const int4*)(g.d_pritems + g.pri_off[level]), ni, ib, Z, XP, RHS, prolong_coeff, S);
}

}  // namespace launch
}  // namespace cirrus
