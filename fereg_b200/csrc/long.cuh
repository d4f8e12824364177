// Kernels for the long lists: segments of more than WT cells or rows (LONG_SEG cells in the
// operator) and coordinate lists of more than PULL_WARP_MAX entries, cut into the tiles of
// tiles.cuh. Every pass is bound by the latency of its gathers, so what these kernels do is keep
// many of them in flight: a warp walks a segment tile on its own, with no barrier of the CTA, and
// reads rows along the row (lane = (row group, column) over floor(32 / columns) groups); a heavy
// segment tile (one that would keep its warp busy when the others are done) and every list tile are
// shared by the warps of a CTA, which meet once per segment or list. The operator's kernels use the
// padded vectors and lane groups of short.cuh. All sums have a fixed order.
#pragma once

#include "short.cuh"

namespace fereg {

constexpr u32 LONG_SEG = 32;  // cells of the longest segment one lane group of k_vseg_apply walks alone
constexpr int LT_WPB = 8;     // warps per CTA
constexpr int LR_WPB = 4;     // of k_ltile_resid (its cells' values take up to 16 KB a warp)
constexpr int LR_COLS = 16;   // columns per launch of k_ltile_resid
// Rows of a segment tile of several segments. Tiles are cut by rows as well as cells: a tile of TILE
// cells holds any number of rows, and a sample of few levels makes few tiles (1e7 rows, 11 columns, a
// warp per tile cut by cells alone: one term of 50 levels, one tile, 1960 ms; a CTA per such tile 449;
// cut by rows, the heavy ones to CTAs, 29. 1e3 levels: 253, 47 and 3.1 ms; 1e5: 3.06, 1.57 and 1.00).
// 128 to 2048 rows measure the same, but for fewer, longer segments (60 of 1,000 rows, 12 columns:
// 138, 142 and 170 us at 128, 512 and 2048); 512 leaves two segments of 250 rows a tile.
constexpr u64 LT_ROWS = 512;
// A tile of more than 1 / LT_SHARE of the long segments' rows is heavy: with fewer such tiles than
// that the chip's warps are not all at work. 1e3 tiles of 5,000 rows: 197 us as heavy ones, 325 as light;
// 4e3 tiles of 100 rows: 138 and 109; 2e3 tiles of 100 rows in eight IRLS steps: 3.54 and 3.46 ms.
constexpr u64 LT_SHARE = 1184;

// Lane = (group g, column c) over a chunk of Rc <= 32 columns.
struct RowLanes {
    int G, g, c;
    bool on;
    __device__ __forceinline__ explicit RowLanes(int Rc) {
        const int lane = int(threadIdx.x & 31u);
        G = 32 / Rc;
        g = lane / Rc;
        c = lane % Rc;
        on = g < G;
    }
    // the groups' values of this lane's column, in group order
    __device__ __forceinline__ double total(double v, int Rc) const {
        double s = 0.0;
        for (int i = 0; i < G; i++) s += __shfl_sync(FULL, v, i * Rc + c);
        return s;
    }
};

// Operator pass 1 on segments of more than LONG_SEG cells: t_s = n1inv_s sum_c W_c u_c, a warp per
// tile, a segment's cells dealt to the lane groups; slices of longer segments write partials.
// 4e4 segments of 50 weighted cells, 4 columns: 43 us with one lane group a segment, 25 by
// tiles, 19 with 256-bit gathers.
template <class T, int L, int NBK, bool WEIGHTED>
__global__ void __launch_bounds__(LT_WPB * 32, 4) k_ltile_apply(DevStruct S, DevWeights W, const T* __restrict__ P,
                                                                int Rv, int j0, int Rc, T* __restrict__ t,
                                                                T* __restrict__ part, int stage) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int G = 32 / L;
    constexpr int NL = NBK < WNB ? NBK : WNB;
    const u32 lane = wlane(), g = lane / L, j = lane % L;
    const bool on = int(4 * j) < Rc;
    const size_t Ru = size_t(Rv);
    const T* Pj = P + j0 + 4 * j;
    if (halted(S)) return;
    T* sp = reinterpret_cast<T*>(smem_raw);
    const int nsm = stage ? int(S.ns_acc) : 0;
    if (nsm) stage_small(sp, P, Ru, j0, Rc, S.ms_acc);
    const T* spj = sp + 4 * j;
    auto total = [&](T v) {
#pragma unroll
        for (int o = L; o < 32; o <<= 1) v += __shfl_xor_sync(FULL, v, o);
        return v;
    };
    const TileSet& ts = S.seg;
    for (u32 tile = blockIdx.x * LT_WPB + wid_in_cta(); tile < ts.n; tile += gridDim.x * LT_WPB) {
        const u32 s0 = ts.k0[tile], s1 = ts.k1[tile], c0 = ts.e0[tile], c1 = ts.e1[tile];
        const int pslot = ts.part[tile];
        for (u32 s = s0; s < s1; s++) {
            const u32 a = max(S.seg_off[s], c0), b = min(S.seg_off[s + 1], c1);
            V4<T> acc{T(0), T(0), T(0), T(0)};
            if (on) {
#pragma unroll 4
                for (u32 c = a + g; c < b; c += G) {
                    u32 k[NL];
#pragma unroll
                    for (int q = 0; q < NL; q++) k[q] = __ldg(S.coord + size_t(q) * S.M + c);
                    const V4<T> u = gather4<NBK, L>(S, k, Pj, Ru, c, spj, nsm, Rc);
                    if constexpr (WEIGHTED) fma4(acc, T(W.cell_w[c]), u);
                    else add4(acc, u);
                }
            }
            acc.a = total(acc.a);
            acc.b = total(acc.b);
            acc.c = total(acc.c);
            acc.d = total(acc.d);
            if (g == 0 && on) {
                if (pslot < 0) {
                    const T n = T(W.n1inv[s]);
                    st4(t + size_t(s) * Ru + j0 + 4 * j, V4<T>{acc.a * n, acc.b * n, acc.c * n, acc.d * n});
                } else {
                    st4(part + size_t(pslot) * Ru + j0 + 4 * j, acc);
                }
            }
        }
    }
}

// Operator pass 2 on long coordinate lists: Y[k] = nr_k P[k] + sum over the cells c of k of
// W_c (sum_{other b} P[coord_b(c)] - t_{s(c)}); slices write partials. A CTA per tile, the entries
// dealt to the lane groups of its warps in turn, the groups' sums added by a butterfly and the warps'
// in order. 1.6e6 entries in 110 lists, 12 columns: 104 us by (slot, column) threads, 41 here
// (466 MB of gathered rows through L2).
template <class T, int L, int NBK, bool WEIGHTED>
__global__ void __launch_bounds__(LT_WPB * 32, 4) k_ltile_pull(DevStruct S, DevWeights W, const T* __restrict__ P,
                                                               const T* __restrict__ t, int Rv, int j0, int Rc,
                                                               T* __restrict__ Y, T* __restrict__ part) {
    __shared__ __align__(16) T red[2][LT_WPB][4 * L];
    constexpr int G = 32 / L;
    constexpr int NO = NBK - 1;
    const u32 lane = wlane(), g = lane / L, j = lane % L, w = wid_in_cta();
    const bool on = int(4 * j) < Rc;
    const size_t Ru = size_t(Rv);
    const u32 no = S.nb - 1;
    const T* Pj = P + j0 + 4 * j;
    const T* tj = t + j0 + 4 * j;
    if (halted(S)) return;
    auto total = [&](T v) {
#pragma unroll
        for (int o = L; o < 32; o <<= 1) v += __shfl_xor_sync(FULL, v, o);
        return v;
    };
    const TileSet& ts = S.pull;
    int par = 0;
    for (u32 tile = blockIdx.x; tile < ts.n; tile += gridDim.x) {
        const u32 k0 = ts.k0[tile], k1 = ts.k1[tile], e0 = ts.e0[tile], e1 = ts.e1[tile];
        const int pslot = ts.part[tile];
        for (u32 k = k0; k < k1; k++, par ^= 1) {
            const u32 a = max(S.pl_off[k], e0), b = min(S.pl_off[k + 1], e1);
            V4<T> acc{T(0), T(0), T(0), T(0)};
            if (on) {
#pragma unroll 4
                for (u32 e = a + w * G + g; e < b; e += LT_WPB * G) {
                    const u32 s = __ldcs(S.pl_seg + e);
                    u32 x[NO > 0 ? NO : 1];
#pragma unroll
                    for (int o = 0; o < NO; o++) x[o] = __ldcs(S.pl_other + size_t(e) * no + o);
                    V4<T> v = ld4cg(tj + size_t(s) * Ru);
                    v.a = -v.a;
                    v.b = -v.b;
                    v.c = -v.c;
                    v.d = -v.d;
#pragma unroll
                    for (int o = 0; o < NO; o++) add4(v, ld4(Pj + size_t(x[o]) * Ru));
                    if constexpr (NBK == WNB)
                        for (u32 o = WNO; o < no; o++) add4(v, ld4(Pj + size_t(S.pl_other[size_t(e) * no + o]) * Ru));
                    if constexpr (WEIGHTED) fma4(acc, T(__ldcs(W.pl_w + e)), v);
                    else add4(acc, v);
                }
            }
            acc.a = total(acc.a);
            acc.b = total(acc.b);
            acc.c = total(acc.c);
            acc.d = total(acc.d);
            if (g == 0) st4s(&red[par][w][4 * j], acc);
            __syncthreads();  // two buffers: the next list's warps write the other one
            if (threadIdx.x < u32(Rc)) {
                const u32 c = threadIdx.x;
                T s = T(0);
#pragma unroll
                for (int i = 0; i < LT_WPB; i++) s += red[par][i][c];
                const size_t o = size_t(k) * Ru + j0 + c;
                if (pslot < 0) Y[o] = T(W.nr[k]) * P[o] + s;
                else part[size_t(pslot) * Ru + j0 + c] = s;
            }
        }
    }
}

// Right-hand side pass 1 on the long segments (no small coordinates summed): b1_s = sum over the rows
// of w v (partials for slices), the CTAs' [sum w v^2, sum w v] per column (cta_part, grid x 2R), and
// the cells' sums (cs, M x R) where the list pass reads those instead of the rows. A warp per tile
// (heavy ones: a CTA), cells dealt to the lane groups, the rows of a cell in order.
// 4e4 segments of 50 cells of 5 rows, 3 columns: 300 us by CTA tiles, 102 here (49 us of
// bytes).
__global__ void __launch_bounds__(LT_WPB * 32) k_ltile_rhs(DevStruct S, DevWeights W, const double* __restrict__ rows,
                                                           int R, int j0, int Rc, double* __restrict__ b1,
                                                           double* __restrict__ part, double* __restrict__ cta_part,
                                                           double* __restrict__ cs) {
    __shared__ double red[2][LT_WPB * 32], team[2][LT_WPB][32];
    constexpr int U = 8;
    const RowLanes L(Rc);
    const size_t Ru = size_t(R);
    const TileSet& ts = S.seg;
    const double* vj = rows + j0 + L.c;
    double q = 0.0, ws = 0.0;
    int par = 0;
    auto take = [&](u32 tile, u32 w, auto warps) {  // warp w of the tile's warps
        constexpr u32 NW = decltype(warps)::value;
        const u32 s0 = ts.k0[tile], s1 = ts.k1[tile], c0 = ts.e0[tile], c1 = ts.e1[tile];
        const int pslot = ts.part[tile];
        const u32 first = w * u32(L.G) + u32(L.g), step = NW * u32(L.G);
        for (u32 s = s0; s < s1; s++) {
            const u32 a = max(S.seg_off[s], c0), b = min(S.seg_off[s + 1], c1);
            double sum = 0.0;
            if (L.on) {
                if (!S.cell_row) {
#pragma unroll 8
                    for (u32 c = a + first; c < b; c += step) {
                        const double v = __ldcs(vj + size_t(c) * Ru);
                        const double wv = W.w_rows ? W.w_rows[c] * v : v;
                        sum += wv;
                        q += wv * v;
                    }
                } else {
                    for (u32 c = a + first; c < b; c += step) {
                        const u32 r0 = S.cell_row[c], r1 = S.cell_row[c + 1];
                        double sc = 0.0;
                        for (u32 r = r0; r < r1; r += U) {
                            double v[U], w[U];
#pragma unroll
                            for (int k = 0; k < U; k++) v[k] = r + k < r1 ? vj[size_t(r + k) * Ru] : 0.0;
#pragma unroll
                            for (int k = 0; k < U; k++) w[k] = (W.w_rows && r + k < r1) ? W.w_rows[r + k] : 1.0;
#pragma unroll
                            for (int k = 0; k < U; k++) {
                                const double wv = w[k] * v[k];
                                sc += wv;
                                q += wv * v[k];
                            }
                        }
                        if (cs) cs[size_t(c) * Ru + j0 + L.c] = sc;
                        sum += sc;
                    }
                }
            }
            ws += sum;
            sum = L.total(sum, Rc);
            if constexpr (NW > 1) {  // the warps in order; two buffers, as in k_ltile_pull
                if (L.on && L.g == 0) team[par][w][L.c] = sum;
                __syncthreads();
                sum = 0.0;
#pragma unroll
                for (u32 i = 0; i < NW; i++) sum += team[par][i][L.c];
                par ^= 1;
            }
            if (w == 0 && L.on && L.g == 0) {
                if (pslot < 0) b1[size_t(s) * Ru + j0 + L.c] = sum;
                else part[size_t(pslot) * Ru + j0 + L.c] = sum;
            }
        }
    };
    using std::integral_constant;
    for (u32 tile = blockIdx.x; tile < ts.nheavy; tile += gridDim.x)
        take(tile, wid_in_cta(), integral_constant<u32, LT_WPB>{});
    for (u32 tile = ts.nheavy + blockIdx.x * LT_WPB + wid_in_cta(); tile < ts.n; tile += gridDim.x * LT_WPB)
        take(tile, 0u, integral_constant<u32, 1>{});
    red[0][threadIdx.x] = q;
    red[1][threadIdx.x] = ws;
    __syncthreads();
    if (int(threadIdx.x) < 2 * Rc) {  // warps and groups in order
        const int h = int(threadIdx.x) / Rc, c = int(threadIdx.x) % Rc;
        double s = 0.0;
        for (int w = 0; w < LT_WPB; w++)
            for (int g = 0; g < L.G; g++) s += red[h][w * 32 + g * Rc + c];
        cta_part[size_t(blockIdx.x) * 2 * Ru + size_t(h) * Ru + j0 + c] = s;
    }
}

// Right-hand side pass 2 on long coordinate lists: rhs[k] = sum over the cells c of k of
// (s_c - W_c b1_{s(c)} / n1_{s(c)}), s_c the sum over the cell's rows (from cs when given); slices
// write partials. A CTA per tile as in k_ltile_pull. 1.6e6 entries, 9 columns: 179 us by (slot,
// column) threads, 59 here.
__global__ void __launch_bounds__(LT_WPB * 32) k_ltile_pull_rhs(DevStruct S, DevWeights W,
                                                                const double* __restrict__ rows,
                                                                const double* __restrict__ b1, int R, int j0, int Rc,
                                                                double* __restrict__ Y, double* __restrict__ part,
                                                                const double* __restrict__ cs) {
    __shared__ double red[2][LT_WPB][32];
    const RowLanes L(Rc);
    const size_t Ru = size_t(R);
    const u32 w = wid_in_cta();
    const TileSet& ts = S.pull;
    const bool direct = cs || !S.cell_row;
    const double* vj = (cs ? cs : rows) + j0 + L.c;
    const double* bj = b1 + j0 + L.c;
    const double* wr = cs ? nullptr : W.w_rows;
    int par = 0;
    for (u32 tile = blockIdx.x; tile < ts.n; tile += gridDim.x) {
        const u32 k0 = ts.k0[tile], k1 = ts.k1[tile], e0 = ts.e0[tile], e1 = ts.e1[tile];
        const int pslot = ts.part[tile];
        for (u32 k = k0; k < k1; k++, par ^= 1) {
            const u32 a = max(S.pl_off[k], e0), b = min(S.pl_off[k + 1], e1);
            double acc = 0.0;
            if (L.on) {
                if (direct) {
#pragma unroll 8
                    for (u32 e = a + w * u32(L.G) + u32(L.g); e < b; e += LT_WPB * u32(L.G)) {
                        const u32 c = __ldcs(S.pl_cell + e), s = __ldcs(S.pl_seg + e);
                        const double x = __ldg(vj + size_t(c) * Ru);
                        const double sc = wr ? wr[c] * x : x;
                        acc += sc - cellw(W, c) * __ldcg(bj + size_t(s) * Ru) * W.n1inv[s];
                    }
                } else {
                    for (u32 e = a + w * u32(L.G) + u32(L.g); e < b; e += LT_WPB * u32(L.G)) {
                        const u32 c = __ldcs(S.pl_cell + e), s = __ldcs(S.pl_seg + e);
                        const u32 re = S.cell_row[c + 1];
                        double sc = 0.0;
#pragma unroll 4
                        for (u32 r = S.cell_row[c]; r < re; r++) {
                            const double x = __ldg(vj + size_t(r) * Ru);
                            sc += wr ? wr[r] * x : x;
                        }
                        acc += sc - cellw(W, c) * __ldcg(bj + size_t(s) * Ru) * W.n1inv[s];
                    }
                }
            }
            acc = L.total(acc, Rc);
            if (L.on && L.g == 0) red[par][w][L.c] = acc;
            __syncthreads();  // two buffers, as above
            if (int(threadIdx.x) < Rc) {
                double s = 0.0;
#pragma unroll
                for (int i = 0; i < LT_WPB; i++) s += red[par][i][threadIdx.x];
                if (pslot < 0) Y[size_t(k) * Ru + j0 + threadIdx.x] = s;
                else part[size_t(pslot) * Ru + j0 + threadIdx.x] = s;
            }
        }
    }
}

// Residualization of the long segments (operator.rs:1107-1179): alpha_s = (b1_s - sum_c W_c u_c) / n1_s
// with u_c = sum_b x[coord_b(c)], then every row of cell c loses alpha_s + u_c. A warp per tile (heavy
// ones: a CTA): the cells' u and first rows into shared memory, alpha of each segment (slices of long segments take it
// from `along`, index fixidx, filled beforehand), then the segment's rows, 8 of them in flight a
// lane. 4e4 segments of 50 cells of 5 rows, 3 columns: 558 us by CTA tiles, 133 here (73 us of
// bytes).
__host__ __device__ constexpr size_t ltile_resid_bytes(int Rc) {
    return al16(size_t(TILE) * Rc * 8) + al16((TILE + 1) * 4);
}
template <int NBK>
__global__ void __launch_bounds__(LR_WPB * 32) k_ltile_resid(DevStruct S, DevWeights W, double* __restrict__ rows,
                                                             int R, int j0, int Rc, const double* __restrict__ x,
                                                             const double* __restrict__ b1,
                                                             const double* __restrict__ along,
                                                             double* __restrict__ alpha) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double team[2][LR_WPB][LR_COLS];
    constexpr int NL = NBK < WNB ? NBK : WNB;
    constexpr int U = 8;
    const RowLanes L(Rc);
    const size_t Ru = size_t(R);
    const u32 lane = wlane(), uRc = u32(Rc);
    const TileSet& ts = S.seg;
    double* vj = rows + j0 + L.c;
    int par = 0;
    auto take = [&](u32 tile, u32 w, unsigned char* mine, auto warps) {  // warp w of the tile's warps
        constexpr u32 NW = decltype(warps)::value;
        auto meet = [&]() {
            if constexpr (NW > 1) __syncthreads();
            else __syncwarp();
        };
        double* us = reinterpret_cast<double*>(mine);
        u32* cr = reinterpret_cast<u32*>(mine + al16(size_t(TILE) * Rc * 8));
        const u32 s0 = ts.k0[tile], s1 = ts.k1[tile], c0 = ts.e0[tile], c1 = ts.e1[tile], nc = c1 - c0;
        const int fidx = ts.fixidx[tile];
        const u32 me = w * 32u + lane, first = w * u32(L.G) + u32(L.g), step = NW * u32(L.G);
        if (S.cell_row)
            for (u32 i = me; i <= nc; i += NW * 32u) cr[i] = S.cell_row[c0 + i];
#pragma unroll 4
        for (u32 e = me; e < nc * uRc; e += NW * 32u) {
            const u32 i = e / uRc, c = e % uRc;
            double u = 0.0;
#pragma unroll
            for (int q = 0; q < NL; q++) u += __ldg(x + size_t(__ldg(S.coord + size_t(q) * S.M + c0 + i)) * Ru + j0 + c);
            if constexpr (NBK == WNB)
                for (u32 q = WNB; q < S.nb; q++) u += __ldg(x + size_t(S.coord[size_t(q) * S.M + c0 + i]) * Ru + j0 + c);
            us[e] = u;
        }
        meet();
        for (u32 s = s0; s < s1; s++) {
            const u32 a = max(S.seg_off[s], c0) - c0, b = min(S.seg_off[s + 1], c1) - c0;
            double al = 0.0;
            if (fidx < 0) {
                double tot = 0.0;
                if (L.on)
                    for (u32 i = a + first; i < b; i += step) tot += cellw(W, c0 + i) * us[i * uRc + L.c];
                tot = L.total(tot, Rc);
                if constexpr (NW > 1) {  // the warps in order; two buffers, as in k_ltile_pull
                    if (L.on && L.g == 0) team[par][w][L.c] = tot;
                    __syncthreads();
                    tot = 0.0;
#pragma unroll
                    for (u32 i = 0; i < NW; i++) tot += team[par][i][L.c];
                    par ^= 1;
                }
                al = (b1[size_t(s) * Ru + j0 + L.c] - tot) * W.n1inv[s];
                if (alpha && w == 0 && L.on && L.g == 0) alpha[size_t(s) * Ru + j0 + L.c] = al;
            } else {
                al = along[size_t(fidx) * Ru + j0 + L.c];
            }
            if (L.on) {
                const u32 r0 = S.cell_row ? cr[a] : c0 + a, r1 = S.cell_row ? cr[b] : c0 + b;
                u32 i = a;
                for (u32 r = r0 + first; r < r1; r += U * step) {
                    double v[U];
#pragma unroll
                    for (int k = 0; k < U; k++) {
                        const u32 rr = r + u32(k) * step;
                        v[k] = rr < r1 ? __ldcs(vj + size_t(rr) * Ru) : 0.0;
                    }
#pragma unroll
                    for (int k = 0; k < U; k++) {
                        const u32 rr = r + u32(k) * step;
                        if (rr < r1) {
                            if (S.cell_row)
                                while (cr[i + 1] <= rr) i++;
                            else i = rr - c0;
                            __stcs(vj + size_t(rr) * Ru, v[k] - (al + us[i * uRc + L.c]));
                        }
                    }
                }
            }
        }
        meet();  // the next tile's values replace these
    };
    using std::integral_constant;
    for (u32 tile = blockIdx.x; tile < ts.nheavy; tile += gridDim.x)
        take(tile, wid_in_cta(), smem_raw, integral_constant<u32, LR_WPB>{});
    unsigned char* own = smem_raw + size_t(wid_in_cta()) * ltile_resid_bytes(Rc);
    for (u32 tile = ts.nheavy + blockIdx.x * LR_WPB + wid_in_cta(); tile < ts.n; tile += gridDim.x * LR_WPB)
        take(tile, 0u, own, integral_constant<u32, 1>{});
}

}  // namespace fereg
