// sm_100a kernels of the fixed-effects solve.
//
// Layout in HBM (one absorber):
//   seg_off[g1+1]       cells of each FE1 level (segment), cells sorted by (FE1, codes, obs)
//   coord[nb*M]         block-major global reduced coordinate of every cell
//   cell_row[M+1]       first row of each cell (absent when every cell holds one row)
//   pl_off[m+1], pl_cell/pl_seg[E], pl_other[E*(nb-1)]
//                       coordinate-sorted cell lists (transpose of coord) with each cell's
//                       segment and other-block coordinates beside it
//   rows[n*R]           the caller's row-major column block (FP64), rows in row order
//   reduced vectors     m x R row-major
//
// Every kernel is deterministic: per-cell values are never scattered; sums by coordinate are
// pulls over the coordinate-sorted lists in list order (tiles.cuh), and column sums combine
// fixed per-CTA partials in CTA order. No floating-point atomics.
#pragma once

#include "long.cuh"
#include "short.cuh"

namespace fereg {

__device__ __forceinline__ int gwarp() { return int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); }
__device__ __forceinline__ int nwarps() { return int((gridDim.x * blockDim.x) >> 5); }
__device__ __forceinline__ int lane_id() { return int(threadIdx.x & 31); }

// ---------------------------------------------------------------------------------------------
// PCG vector work on m x R blocks (cg.rs), column sums as per-CTA partials (gridDim x R).
template <class T>
__global__ void __launch_bounds__(TB) k_dot(const T* __restrict__ a, const T* __restrict__ b, u32 m, int R,
                                            double* __restrict__ cta_part) {
    __shared__ double red[TB];
    for (int j0 = 0; j0 < R; j0 += RC_MAX) {
        const ColMap cm = colmap(R, j0);
        double acc = 0.0;
        if (cm.on)
            for (u32 i = blockIdx.x * u32(cm.nslot) + u32(cm.slot); i < m; i += gridDim.x * u32(cm.nslot)) {
                const size_t o = size_t(i) * R + j0 + cm.col;
                acc += double(a[o]) * double(b[o]);
            }
        red[threadIdx.x] = acc;
        __syncthreads();
        if (int(threadIdx.x) < cm.Rc) {
            double s = 0.0;
            for (int sl = 0; sl < cm.nslot; sl++) s += red[sl * cm.Rc + threadIdx.x];
            cta_part[size_t(blockIdx.x) * R + j0 + threadIdx.x] = s;
        }
        __syncthreads();
    }
}

// Column sums of [nparts x ncols] partials (plus a second array when given) in a fixed order:
// one warp per column, lane l sums parts l, l+32, ..., then a fixed butterfly.
__global__ void k_reduce_cols(const double* __restrict__ part, int nparts, const double* __restrict__ part2,
                              int nparts2, int ncols, double* __restrict__ out) {
    const int lane = lane_id();
    for (int col = gwarp(); col < ncols; col += nwarps()) {
        double acc = 0.0;
        for (int p = lane; p < nparts; p += 32) acc += part[size_t(p) * ncols + col];
        if (part2)
            for (int p = lane; p < nparts2; p += 32) acc += part2[size_t(p) * ncols + col];
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
        if (lane == 0) out[col] = acc;
    }
}

// The same sums of one array of many parts (a part per level of a term): a CTA per column, so that a
// column's chain of loads is short. 2e4 parts of 9 columns: 168 us by warps, 8 here.
constexpr int TALL_TB = 1024, TALL_PARTS = 4096;
__global__ void __launch_bounds__(TALL_TB) k_reduce_tall(const double* __restrict__ part, int nparts, int ncols,
                                                         double* __restrict__ out) {
    __shared__ double red[TALL_TB / 32];
    for (int col = blockIdx.x; col < ncols; col += gridDim.x) {
        double acc = 0.0;
#pragma unroll 8
        for (int p = threadIdx.x; p < nparts; p += TALL_TB) acc += part[size_t(p) * ncols + col];
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
        if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < TALL_TB / 32; w++) t += red[w];
            out[col] = t;
        }
        __syncthreads();
    }
}

// Per-column PCG state (cg.rs:132-292), kept on the device. active: 1 iterating, 0 stopped by
// the reference's rules, 2 stopped at the FP32 precision floor of a refinement round.
struct CgState {
    double* rho;
    double* pq;
    double* gamma;
    double* beta;
    double* xb;      // d'rhs, d'r, x0'r (3R)
    double* ss1;
    double* floor_;  // 1e-26 * ss0
    double* ring;    // R x WINDOW
    double* xconst;  // x0'rhs
    double* pfloor;  // precision floor of the preconditioned residual (0: none)
    int* active;
    int* n_active;
};

constexpr int WINDOW = 5;

// End of an FP32 refinement round, on the FP64 quantities of the refined iterate x: rho = r'M^-1 r
// of its true residual, xconst = x'rhs, pq = x'r. A column is accepted (state 0) only when
// rho <= max(tol^2 ss_k, floor) with ss_k = ss1 - x'(rhs + r), whether the round ended it by the
// FP32 window rule (whose recursive residual can fall below the true one) or at the FP32 floor;
// otherwise it goes another round (state 1). Columns without variation (floor 0) stay stopped.
__global__ void k_refine_accept(CgState st, int R, double tol) {
    __shared__ int cnt;
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    int local = 0;
    for (int j = threadIdx.x; j < R; j += blockDim.x) {
        if (st.floor_[j] > 0.0) {
            const double ssk = st.ss1[j] - (st.xconst[j] + st.pq[j]);
            const double thr = fmax(tol * tol * ssk, st.floor_[j]);
            const bool ok = st.rho[j] <= thr;
            st.active[j] = ok ? 0 : 1;
        }
        local += st.active[j] == 1;
    }
    atomicAdd(&cnt, local);  // integer count: order independent
    __syncthreads();
    if (threadIdx.x == 0) *st.n_active = cnt;
}

template <class Src, class Dst>
__global__ void k_convert(const Src* __restrict__ a, Dst* __restrict__ b, size_t total) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x)
        b[i] = Dst(a[i]);
}

// x += d (the FP32 correction of a refinement round).
__global__ void k_add_correction(double* __restrict__ x, const float* __restrict__ d, size_t total) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x)
        x[i] += double(d[i]);
}

// r = a - b
template <class T>
__global__ void k_sub(T* __restrict__ r, const T* __restrict__ a, const T* __restrict__ b, size_t total) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x)
        r[i] = a[i] - b[i];
}

// x = 0 on the columns whose mask is 1 (warm starts of zero columns, solve.rs:1209-1217).
__global__ void k_zero_masked(double* __restrict__ x, const int* __restrict__ mask, size_t total, int R) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x)
        if (mask[i % R]) x[i] = 0.0;
}

// The solve's column scalars from the rhs pass's column sums cs = [sum w v^2, sum w v, sum b1^2/n1]
// (solve.rs:1210-1217): ss0 = the weighted centered sum of squares (0 below 1e-15 of the sum of
// squares), ss1 = sum w v^2 - sum b1^2/n1, and the PCG's start state: active = ss0 > 0, the floor
// 1e-26 ss0, x'rhs of the start 0. Columns r..rv-1 (padding) get zeros.
__global__ void k_ss_prep(const double* __restrict__ cs, int r, int rv, double sw, double* __restrict__ ss0,
                          double* __restrict__ ss1, int* __restrict__ active, double* __restrict__ floor_,
                          double* __restrict__ xconst) {
    for (int j = int(blockIdx.x * blockDim.x + threadIdx.x); j < rv; j += int(gridDim.x * blockDim.x)) {
        double s0 = 0.0, s1 = 0.0;
        if (j < r) {
            const double wsq = cs[j], wsum = cs[r + j], b1sq = cs[2 * r + j];
            const double s = wsq - wsum * wsum / sw;
            s0 = s > 1e-15 * wsq ? s : 0.0;
            s1 = wsq - b1sq;
        }
        ss0[j] = s0;
        ss1[j] = s1;
        active[j] = s0 > 0.0;
        floor_[j] = 1e-26 * s0;
        xconst[j] = 0.0;
    }
}

// x = 0 on the columns j < r whose ss0 is 0 (a warm start of zero columns, solve.rs:1209-1217).
__global__ void k_zero_ss0(double* __restrict__ x, const double* __restrict__ ss0, size_t total, int R, int r) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
        const int j = int(i % size_t(R));
        if (j < r && ss0[j] == 0.0) x[i] = 0.0;
    }
}

// x += z on the active columns (exact preconditioner, cg.rs:171-198).
template <class T>
__global__ void k_add_active(T* __restrict__ x, const T* __restrict__ z, const int* __restrict__ active, size_t total, int R) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x)
        if (active[i % R] == 1) x[i] += z[i];
}

// The small coordinates' rows of Y = S P from the dense rows of S (srow, weights.cuh): CTA b
// takes the coordinates f of its chunk; with at most TB (k, j) pairs the threads are (slot, pair)
// and slot s adds srow[f][k] P[f][j] over the chunk's f = s, s + slots, ... (loads unrolled),
// the slots' sums are then added in slot order into part[b][k * R + j]; with more pairs each
// thread takes pairs in turn over the whole chunk. k_small_reduce adds the CTAs' partials in CTA
// order.
template <class T>
__global__ void __launch_bounds__(TB) k_srow_apply(const double* __restrict__ srow, u32 m, u32 ms,
                                                    const T* __restrict__ P, int R, T* __restrict__ part,
                                                    const int* halt) {
    __shared__ T red[TB];
    if (halt && __ldcg(halt)) return;  // the PCG loop has ended (pcg.cuh)
    const u32 npairs = ms * u32(R);
    const u32 chunk = (m + gridDim.x - 1) / gridDim.x;
    const u32 f0 = min(m, blockIdx.x * chunk), f1 = min(m, f0 + chunk);
    if (npairs <= u32(TB)) {
        const u32 nslot = u32(TB) / npairs, slot = threadIdx.x / npairs, pi = threadIdx.x % npairs;
        const u32 k = pi / u32(R), j = pi % u32(R);
        T acc = T(0);
        if (slot < nslot) {
#pragma unroll 4
            for (u32 f = f0 + slot; f < f1; f += nslot) acc += T(srow[size_t(f) * ms + k]) * P[size_t(f) * R + j];
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        if (threadIdx.x < npairs) {
            T sum = T(0);
            for (u32 sl = 0; sl < nslot; sl++) sum += red[sl * npairs + threadIdx.x];
            part[size_t(blockIdx.x) * npairs + threadIdx.x] = sum;
        }
        return;
    }
    for (u32 pi = threadIdx.x; pi < npairs; pi += blockDim.x) {
        const u32 k = pi / u32(R), j = pi % u32(R);
        T acc = T(0);
#pragma unroll 4
        for (u32 f = f0; f < f1; f++) acc += T(srow[size_t(f) * ms + k]) * P[size_t(f) * R + j];
        part[size_t(blockIdx.x) * npairs + pi] = acc;
    }
}

// Jacobi on coordinates [k0, m): z = inv_diag .* r (precond/jacobi.rs:12-42).
template <class T>
__global__ void k_jacobi(const T* __restrict__ r, T* __restrict__ z, const double* __restrict__ inv_diag, u32 k0, u32 m, int R) {
    const size_t total = size_t(m - k0) * R;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
        const size_t o = size_t(k0) * R + i;
        z[o] = T(inv_diag[k0 + i / R]) * r[o];
    }
}

// Small super-block: z[0..ms) = Minv r[0..ms) with the expanded, scaled generalized inverse.
// z = minv r on the small coordinates (ms x R), one warp per output element: lane l adds the
// products of entries l, l + 32, ... in order, combined by a fixed butterfly.
template <class T>
__global__ void k_small_apply(const double* __restrict__ minv, u32 ms, const T* __restrict__ r, T* __restrict__ z, int R) {
    const size_t total = size_t(ms) * R;
    const u32 lane = threadIdx.x % 32;
    const size_t nw = size_t(gridDim.x) * blockDim.x / 32;
    for (size_t i = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; i < total; i += nw) {
        const u32 row = u32(i / R);
        const int col = int(i % R);
        const double* mr = minv + size_t(row) * ms;
        double acc = 0.0;
        for (u32 l = lane; l < ms; l += 32) acc += mr[l] * double(r[size_t(l) * R + col]);
#pragma unroll
        for (int o = 16; o > 0; o /= 2) acc += __shfl_xor_sync(FULL, acc, o);
        if (lane == 0) z[i] = T(acc);
    }
}

// ---------------------------------------------------------------------------------------------
// Grounded LDL^T of the unit-diagonal-scaled small block (precond/dense.rs:26-38, 79-100): a
// pivot at or below PIVOT_TOL is replaced by GROUND. `a` is k x k row-major and only its lower
// triangle is read; its strict lower part becomes the unit-lower factor L, its strict upper part
// L^T (for the inverse's backward pass), `d` the pivots. Blocked right-looking: a panel of NB
// columns is factored by one CTA in shared memory (k_ldlt_panel), then every CTA of
// k_ldlt_trail subtracts the panel's rank-NB update from one 32 x 32 tile of the trailing lower
// triangle. Column by column the arithmetic is the unblocked one (a[i][l] -= a[i][j] a[l][j] / d_j
// with the pivots taken in order); only the order of the trailing sums differs.
constexpr double PIVOT_TOL = 1e-10;
constexpr double GROUND = 1e30;

// The panel of a block of at most 1024 rows: thread t holds the panel elements of row t in registers,
// the pivot rows' current column passes through shared memory, one barrier per column, the divisions
// by the first warp alone. k = 910: the panel in shared memory with a division per element and two
// barriers a column 59 us, here 19 us.
template <int NB>
__global__ void __launch_bounds__(1024) k_ldlt_panel(double* __restrict__ a, double* __restrict__ d, int k, int jb) {
    __shared__ double top[2][NB], piv[2];
    const int nb = min(NB, k - jb), rows = k - jb, r = int(threadIdx.x);
    double p[NB];
#pragma unroll
    for (int c = 0; c < NB; c++) p[c] = (r < rows && c < nb && r >= c) ? a[size_t(jb + r) * k + jb + c] : 0.0;
#pragma unroll
    for (int jj = 0; jj < NB; jj++) {
        if (jj < nb) {
            // the pivot rows divide; the others would spend the FP64 pipe on the same quotients
            if (r < 32) {
                double dj = __shfl_sync(FULL, p[jj], jj);
                if (dj <= PIVOT_TOL) dj = GROUND;
                if (r == 0) {
                    d[jb + jj] = dj;
                    piv[jj & 1] = 1.0 / dj;
                }
                if (r < NB) top[jj & 1][r] = p[jj] / dj;
            }
            __syncthreads();
            const double inv = piv[jj & 1], m = p[jj];
#pragma unroll
            for (int l = jj + 1; l < NB; l++)
                if (l < nb) p[l] -= m * top[jj & 1][l];
            if (r > jj) p[jj] = m * inv;  // L
        }
    }
#pragma unroll
    for (int c = 0; c < NB; c++)
        if (r < rows && c < nb && r > c) {
            a[size_t(jb + r) * k + jb + c] = p[c];
            a[size_t(jb + c) * k + jb + r] = p[c];
        }
}

// The panel in shared memory with a division per element: the rounding of the blocks that keep it
// (dense_ldlt_inverse).
template <int NB>
__global__ void __launch_bounds__(1024) k_ldlt_panel_div(double* __restrict__ a, double* __restrict__ d, int k, int jb) {
    extern __shared__ double P[];  // rows jb..k-1 of the panel columns jb..jb+NB-1, NB per row
    const int nb = min(NB, k - jb), rows = k - jb;
    for (int idx = threadIdx.x; idx < rows * NB; idx += blockDim.x) {
        const int r = idx / NB, c = idx % NB;
        P[idx] = (c < nb && r >= c) ? a[size_t(jb + r) * k + jb + c] : 0.0;
    }
    for (int jj = 0; jj < nb; jj++) {
        __syncthreads();
        double dj = P[jj * NB + jj];
        if (dj <= PIVOT_TOL) dj = GROUND;
        if (threadIdx.x == 0) d[jb + jj] = dj;
        // the panel's later columns: P[r][l] -= P[r][jj] P[l][jj] / dj for jj < l <= r
        for (int idx = threadIdx.x; idx < (rows - jj - 1) * NB; idx += blockDim.x) {
            const int r = jj + 1 + idx / NB, l = idx % NB;
            if (l > jj && l < nb && l <= r) P[r * NB + l] -= P[r * NB + jj] * P[l * NB + jj] / dj;
        }
        __syncthreads();
        for (int r = jj + 1 + int(threadIdx.x); r < rows; r += blockDim.x) P[r * NB + jj] /= dj;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < rows * NB; idx += blockDim.x) {
        const int r = idx / NB, c = idx % NB;
        if (c < nb && r > c) {
            a[size_t(jb + r) * k + jb + c] = P[idx];
            a[size_t(jb + c) * k + jb + r] = P[idx];
        }
    }
}

// The whole factor by one CTA for k up to LDLT_WHOLE, without a launch per panel: thread (x, y)
// holds the elements (y + 16 p, x + 16 q) of what is left of the matrix in registers, the current
// column passes through shared memory, one barrier and one reciprocal per column. After 16 columns
// the finished block column is written out and the registers move up one block, so that one body
// serves every column (a body per block column took 40 us at k = 110 with its code in the
// instruction cache and 90 us without). 256 threads: with 1024 the FP64 pipe spends more on
// reciprocals than on products (67 us). By panels 111 us, here 43 us.
constexpr int LDLT_WHOLE = 160;
template <int NR>  // k <= 16 NR
__global__ void __launch_bounds__(256) k_ldlt_whole(double* __restrict__ a, double* __restrict__ d, int k) {
    __shared__ double col[2][16 * NR], rec[16];
    const int x = int(threadIdx.x % 16), y = int(threadIdx.x / 16);
    double e[NR][NR];
#pragma unroll
    for (int p = 0; p < NR; p++)
#pragma unroll
        for (int q = 0; q <= p; q++) {
            const int r = y + 16 * p, c = x + 16 * q;
            e[p][q] = (r < k && c <= r) ? a[size_t(r) * k + c] : 0.0;
        }
    for (int b = 0; b < k; b += 16) {
        const int n = k - b;  // rows left
        for (int j = 0; j < min(16, n); j++) {
            double* cj = col[j & 1];
            if (x == j) {
#pragma unroll
                for (int p = 0; p < NR; p++) cj[y + 16 * p] = e[p][0];
            }
            __syncthreads();
            double dj = cj[j];
            if (dj <= PIVOT_TOL) dj = GROUND;
            const double inv = 1.0 / dj;
            if (threadIdx.x == 0) {
                d[b + j] = dj;
                rec[j] = inv;
            }
            // 0 in the finished columns and rows, which keep their values; no branch on the blocks
            // left, which would serialize the loads
            double f[NR], m[NR];
#pragma unroll
            for (int q = 0; q < NR; q++) {
                f[q] = cj[x + 16 * q] * inv;
                m[q] = cj[y + 16 * q];
            }
            if (x <= j) f[0] = 0.0;
            if (y <= j) m[0] = 0.0;
#pragma unroll
            for (int p = 0; p < NR; p++)
#pragma unroll
                for (int q = 0; q <= p; q++) e[p][q] -= m[p] * f[q];
        }
        __syncthreads();
        const double ri = rec[x];
#pragma unroll
        for (int p = 0; p < NR; p++) {
            const int r = y + 16 * p;
            if (r < n && r > x && x < n) a[size_t(b + r) * k + b + x] = a[size_t(b + x) * k + b + r] = e[p][0] * ri;
        }
        __syncthreads();  // rec is written again
#pragma unroll
        for (int p = 0; p + 1 < NR; p++)
#pragma unroll
            for (int q = 0; q <= p; q++) e[p][q] = e[p + 1][q + 1];
#pragma unroll
        for (int q = 0; q < NR; q++) e[NR - 1][q] = 0.0;
    }
}

// Tile (ti, tl), tl <= ti, of the trailing lower triangle (rows and columns from jb + nb): a[i][l]
// -= sum over the panel's columns p of L[i][p] d_p L[l][p], for l <= i.
template <int NB>
__global__ void __launch_bounds__(256) k_ldlt_trail(double* __restrict__ a, const double* __restrict__ d, int k, int jb,
                                                    int nb) {
    __shared__ double Li[32][NB + 1], Ll[32][NB + 1];
    const int t0 = jb + nb, b = int(blockIdx.x);
    int ti = int((sqrt(8.0 * b + 1.0) - 1.0) / 2.0);
    while ((ti + 1) * (ti + 2) / 2 <= b) ti++;
    while (ti * (ti + 1) / 2 > b) ti--;
    const int tl = b - ti * (ti + 1) / 2;
    const int i0 = t0 + 32 * ti, l0 = t0 + 32 * tl;
    for (int idx = threadIdx.x; idx < 32 * NB; idx += blockDim.x) {
        const int r = idx / NB, p = idx % NB;
        Li[r][p] = (i0 + r < k && p < nb) ? a[size_t(i0 + r) * k + jb + p] : 0.0;
        Ll[r][p] = (l0 + r < k && p < nb) ? a[size_t(l0 + r) * k + jb + p] * d[jb + p] : 0.0;
    }
    __syncthreads();
    const int tx = int(threadIdx.x % 32), ty = int(threadIdx.x / 32);
    const int l = l0 + tx;
    for (int rr = ty; rr < 32; rr += int(blockDim.x / 32)) {
        const int i = i0 + rr;
        if (i < k && l < k && l <= i) {
            double s = 0.0;
#pragma unroll
            for (int p = 0; p < NB; p++) s += Li[rr][p] * Ll[tx][p];
            a[size_t(i) * k + l] -= s;
        }
    }
}

// X = L^-T D^-1 L^-1 for k up to 32 NR, one warp per NC columns of X, the columns in registers (lane
// l holds the rows l, l + 32, ...). Column-oriented: once v[p] is final every lane subtracts its
// rows' multiples of it, so a step costs one shuffle and one product on the chain, and the rows of
// L of the next U steps are in flight meanwhile. What bounds it is that chain (small k) and the
// matrix's passes through L2, which NC = 2 halves (large k). Against the row-oriented form with a
// warp-wide sum per row: k = 110 114 -> 17 us, k = 310 422 -> 102 us, k = 910 2039 -> 576 us.
template <int NR, int NC>
__global__ void __launch_bounds__(128) k_ldlt_inverse(const double* __restrict__ a, const double* __restrict__ d, int k,
                                                      double* __restrict__ x) {
    constexpr int U = NR >= 32 ? 1 : NR >= 16 ? 2 : 8;
    const int lane = int(threadIdx.x % 32);
    const int col = (int(blockIdx.x) * 4 + int(threadIdx.x / 32)) * NC;
    if (col >= k) return;  // whole warps
    double v[NC][NR];
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
        for (int r = 0; r < NR; r++) v[c][r] = lane + 32 * r == col + c ? 1.0 : 0.0;
    // forward: v[i] -= L[i][p] v[p], i > p (row p of the upper triangle is L's column p)
#pragma unroll
    for (int q = 0; q < NR; q++) {
        if (32 * q + 31 < col || 32 * q >= k) continue;
        for (int l0 = 0; l0 < 32; l0 += U) {
            double row[U][NR];
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int r = q; r < NR; r++) {
                    const int p = 32 * q + l0 + u, i = lane + 32 * r;
                    row[u][r] = (p < i && i < k) ? a[size_t(p) * k + i] : 0.0;
                }
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const double vp = __shfl_sync(FULL, v[c][q], l0 + u);
#pragma unroll
                    for (int r = q; r < NR; r++) v[c][r] -= row[u][r] * vp;
                }
        }
    }
#pragma unroll
    for (int r = 0; r < NR; r++)
        if (lane + 32 * r < k) {
            const double dr = d[lane + 32 * r];
#pragma unroll
            for (int c = 0; c < NC; c++) v[c][r] /= dr;
        }
    // backward: v[i] -= L[p][i] v[p], i < p (row p of the lower triangle)
#pragma unroll
    for (int q = NR - 1; q >= 0; q--) {
        if (32 * q >= k) continue;
        for (int l0 = 32 - U; l0 >= 0; l0 -= U) {
            double row[U][NR];
#pragma unroll
            for (int u = U - 1; u >= 0; u--)
#pragma unroll
                for (int r = 0; r <= q; r++) {
                    const int p = 32 * q + l0 + u, i = lane + 32 * r;
                    row[u][r] = (p < k && i < p) ? a[size_t(p) * k + i] : 0.0;
                }
#pragma unroll
            for (int u = U - 1; u >= 0; u--)
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const double vp = __shfl_sync(FULL, v[c][q], l0 + u);
#pragma unroll
                    for (int r = 0; r <= q; r++) v[c][r] -= row[u][r] * vp;
                }
        }
    }
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
        for (int r = 0; r < NR; r++)
            if (lane + 32 * r < k && col + c < k) x[size_t(lane + 32 * r) * k + col + c] = v[c][r];
}

// The same by rows, past 1024 rows (the registers do not hold a column) and for the blocks that keep
// its rounding (dense_ldlt_inverse): one warp per column of X (8 per
// block), the column held in shared memory:
// forward over L's rows (strict lower part), the pivots, backward over L^T's rows (strict upper
// part), each step a warp-wide dot product combined by a fixed butterfly.
__global__ void __launch_bounds__(256) k_ldlt_inverse_rows(const double* __restrict__ a, const double* __restrict__ d, int k,
                                                      double* __restrict__ x) {
    extern __shared__ double xs[];
    const int w = int(threadIdx.x / 32), lane = int(threadIdx.x % 32);
    const int col = int(blockIdx.x) * 8 + w;
    if (col >= k) return;  // whole warps
    double* v = xs + size_t(w) * k;
    for (int i = lane; i < k; i += 32) v[i] = i == col ? 1.0 : 0.0;
    __syncwarp();
    for (int i = col + 1; i < k; i++) {
        const double* Li = a + size_t(i) * k;
        double s = 0.0;
        for (int p = col + lane; p < i; p += 32) s += Li[p] * v[p];
#pragma unroll
        for (int o = 16; o > 0; o /= 2) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) v[i] = -s;
        __syncwarp();
    }
    for (int i = lane; i < k; i += 32) v[i] /= d[i];
    __syncwarp();
    for (int i = k - 2; i >= 0; i--) {
        const double* Ui = a + size_t(i) * k;
        double s = 0.0;
        for (int p = i + 1 + lane; p < k; p += 32) s += Ui[p] * v[p];
#pragma unroll
        for (int o = 16; o > 0; o /= 2) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) v[i] -= s;
        __syncwarp();
    }
    for (int i = lane; i < k; i += 32) x[size_t(i) * k + col] = v[i];
}

// minv (ms x ms, zero outside the kept coordinates) = S^-1 X S^-1 scattered to the kept rows/cols.
__global__ void k_expand_minv(const double* __restrict__ x, const u32* __restrict__ keep, const double* __restrict__ scale,
                              int k, u32 ms, double* __restrict__ minv) {
    const size_t total = size_t(k) * k;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
        const int a = int(i / k), b = int(i % k);
        minv[size_t(keep[a]) * ms + keep[b]] = scale[a] * x[i] * scale[b];
    }
}

}  // namespace fereg
