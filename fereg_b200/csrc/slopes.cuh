// Device passes of the heterogeneous-slope absorber (slopes.h): the segment pass over the
// levels of the eliminated term E (slopes.rs:1025-1137 seg_task, 1161-1262 resid_task), the
// coordinate pass over the coordinate-sorted slot lists, and the block-Jacobi preconditioner
// (slopes.rs:1996 SPre::apply on its Jacobi blocks). Every sum has a fixed order.
#pragma once

#include "vec4.cuh"

namespace fereg {

constexpr int SL_BE_MAX = 8;  // width (intercept + slopes) of the eliminated term
constexpr int SL_B_MAX = 8;   // width of the other terms
constexpr int SL_TB = 256;

struct SlopeDev {
    u32 n, ge, k, m, be, e_ns;
    int e_icpt;
    const u32* seg_off;  // ge + 1
    const u32* sc;       // n x k
    const double* sv;    // n x k
    const double* he;    // n x e_ns
    const double* w;     // n, or null (1)
    const double* minv;  // ge x be^2
};

enum SlMode { SL_RHS = 1, SL_RESID = 2 };

// Design value l of E in row i: (1?, slopes...).
__device__ __forceinline__ double sl_he(const SlopeDev& D, u32 i, int l) {
    if (D.e_icpt) return l == 0 ? 1.0 : D.he[size_t(i) * D.e_ns + (l - 1)];
    return D.he[size_t(i) * D.e_ns + l];
}

// The loaded value of row i in column j: RHS the row (src, n x lds); RESID d_i = v_i - u_i(x) with
// u_i = sum_slots v x[c] (x: m x ldx, or null when m = 0).
template <int MODE>
__device__ __forceinline__ double sl_load(const SlopeDev& D, u32 i, int j, const double* __restrict__ src, int lds,
                                          const double* __restrict__ x, int ldx) {
    if constexpr (MODE == SL_RHS) {
        return src[size_t(i) * lds + j];
    } else {
        double u = 0.0;
        if (x)
            for (u32 t = 0; t < D.k; t++) {
                const size_t e = size_t(i) * D.k + t;
                u += D.sv[e] * x[size_t(D.sc[e]) * ldx + j];
            }
        return src[size_t(i) * lds + j] - u;
    }
}

// The segment pass over levels s of E and columns j < C, once each in a solve, a thread per (level,
// column):
//   t = M_s^+ sum_i w_i h_E,i y_i,  e_i = y_i - h_E,i' t,
// RHS: Z[i, j] = w_i e_i (n x ldz) and the per-level partials [sum w y^2, sum w y, sum w e^2]
// (part: ge x 3C); RESID: the row becomes e_i (in place) and alpha[s be + l, j] = t_l.
template <int MODE>
__global__ void __launch_bounds__(SL_TB) k_sl_seg(SlopeDev D, const double* src, int lds, int C,
                                                   const double* __restrict__ x, int ldx, double* __restrict__ Z,
                                                   int ldz, double* rows_out, double* __restrict__ alpha, int lda,
                                                   double* __restrict__ part) {
    const size_t total = size_t(D.ge) * C;
    const int be = int(D.be);
    for (size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q < total; q += size_t(gridDim.x) * blockDim.x) {
        const u32 s = u32(q / C);
        const int j = int(q % C);
        const u32 r0 = D.seg_off[s], r1 = D.seg_off[s + 1];
        double a[SL_BE_MAX], t[SL_BE_MAX];
#pragma unroll
        for (int l = 0; l < SL_BE_MAX; l++) a[l] = 0.0;
        double swv2 = 0.0, swv = 0.0, swe2 = 0.0;
        for (u32 i = r0; i < r1; i++) {
            const double y = sl_load<MODE>(D, i, j, src, lds, x, ldx);
            const double wi = D.w ? D.w[i] : 1.0;
#pragma unroll
            for (int l = 0; l < SL_BE_MAX; l++)
                if (l < be) a[l] += wi * sl_he(D, i, l) * y;
            if constexpr (MODE == SL_RHS) {
                swv2 += wi * y * y;
                swv += wi * y;
            }
        }
        const double* mv = D.minv + size_t(s) * be * be;
#pragma unroll
        for (int l = 0; l < SL_BE_MAX; l++) {
            double v = 0.0;
            if (l < be)
                for (int l2 = 0; l2 < be; l2++) {
                    const double c = mv[l * be + l2];
                    if (c != 0.0) v += c * a[l2];
                }
            t[l] = v;
        }
        for (u32 i = r0; i < r1; i++) {
            const double y = sl_load<MODE>(D, i, j, src, lds, x, ldx);
            double e = y;
#pragma unroll
            for (int l = 0; l < SL_BE_MAX; l++)
                if (l < be) e -= sl_he(D, i, l) * t[l];
            if constexpr (MODE == SL_RESID) {
                rows_out[size_t(i) * lds + j] = e;
            } else {
                const double wi = D.w ? D.w[i] : 1.0;
                Z[size_t(i) * ldz + j] = wi * e;
                if constexpr (MODE == SL_RHS) swe2 += wi * e * e;
            }
        }
        if constexpr (MODE == SL_RESID) {
            if (alpha)
                for (int l = 0; l < be; l++) alpha[(size_t(s) * be + l) * lda + j] = t[l];
        }
        if constexpr (MODE == SL_RHS) {
            double* pp = part + size_t(s) * 3 * C;
            pp[j] = swv2;
            pp[C + j] = swv;
            pp[2 * C + j] = swe2;
        }
    }
}

// The segment pass of the operator, y_i = u_i = sum_slots v P[c] (P: m x R, R a multiple of 4): a group
// of GL lanes per level and four columns, lane i holding row i of the level, whose value stays in
// registers for the second walk where the level has at most GL rows; the lanes' products are summed
// by a fixed butterfly. Gathers of P and a short serial chain bound it: 2e5 rows, 2e4 levels, 4
// columns 14.5 us by a thread per (level, column), 6.1 here. BE: the width of E at most.
template <int BE, int GL>
__global__ void __launch_bounds__(SL_TB) k_sl_apply(SlopeDev D, const double* __restrict__ P, int R,
                                                    double* __restrict__ Z, const int* halt) {
    if (halt && __ldcg(halt)) return;  // the PCG loop has ended (pcg.cuh)
    const u32 lane = threadIdx.x % GL, wl = threadIdx.x & 31u;
    const unsigned gmask = GL == 32 ? 0xffffffffu : ((1u << (GL % 32)) - 1u) << (wl / GL * GL);
    const u32 Q = u32(R) / 4, be = D.be;
    const size_t total = size_t(D.ge) * Q, step = size_t(gridDim.x) * (SL_TB / GL);
    for (size_t q = (size_t(blockIdx.x) * SL_TB + threadIdx.x) / GL; q < total; q += step) {
        const u32 s = u32(q / Q);
        const size_t j = 4 * (q % Q);
        const u32 r0 = D.seg_off[s], r1 = D.seg_off[s + 1];
        auto u_of = [&](u32 i) {
            V4<double> u{0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
            for (u32 t = 0; t < D.k; t++) {
                const size_t e = size_t(i) * D.k + t;
                fma4(u, D.sv[e], ld4(P + size_t(D.sc[e]) * R + j));
            }
            return u;
        };
        V4<double> a[BE], t[BE], y{0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int l = 0; l < BE; l++) a[l] = t[l] = V4<double>{0.0, 0.0, 0.0, 0.0};
        for (u32 i = r0 + lane; i < r1; i += GL) {
            y = u_of(i);
            const double wi = D.w ? D.w[i] : 1.0;
#pragma unroll
            for (int l = 0; l < BE; l++)
                if (l < int(be)) fma4(a[l], wi * sl_he(D, i, l), y);
        }
#pragma unroll
        for (int l = 0; l < BE; l++)
            if (l < int(be))
#pragma unroll
                for (int o = GL / 2; o > 0; o >>= 1) {
                    a[l].a += __shfl_xor_sync(gmask, a[l].a, o, GL);
                    a[l].b += __shfl_xor_sync(gmask, a[l].b, o, GL);
                    a[l].c += __shfl_xor_sync(gmask, a[l].c, o, GL);
                    a[l].d += __shfl_xor_sync(gmask, a[l].d, o, GL);
                }
        const double* mv = D.minv + size_t(s) * be * be;
#pragma unroll
        for (int l = 0; l < BE; l++)
            if (l < int(be))
#pragma unroll
                for (int l2 = 0; l2 < BE; l2++)
                    if (l2 < int(be)) {
                        const double c = mv[u32(l) * be + u32(l2)];
                        if (c != 0.0) fma4(t[l], c, a[l2]);
                    }
        const bool kept = r1 - r0 <= u32(GL);
        for (u32 i = r0 + lane; i < r1; i += GL) {
            V4<double> e = kept ? y : u_of(i);
#pragma unroll
            for (int l = 0; l < BE; l++)
                if (l < int(be)) fma4(e, -sl_he(D, i, l), t[l]);
            const double wi = D.w ? D.w[i] : 1.0;
            st4(Z + size_t(i) * R + j, V4<double>{wi * e.a, wi * e.b, wi * e.c, wi * e.d});
        }
    }
}

// The coordinate pass: Y[c, j] = sum over the list of coordinate c of v Z[row, j], c < m, j < C; Z's
// stride is a multiple of 4 (its columns past C are read and not used). NT lanes per coordinate and
// four columns, entry i, i + NT, ... to lane i, the lanes' sums by a fixed butterfly, the warps' in
// order. A chain of gathers bounds it: lists of 100 rows, 4e3 coordinates, 4 columns 25 us by a
// thread per (coordinate, column), 4.5 by warps (NT = 32); lists of more than SL_LONG entries on
// average take a CTA each (NT = SL_TB).
constexpr u32 SL_LONG = 512;
template <int NT>
__global__ void __launch_bounds__(SL_TB) k_sl_pull(u32 m, int C, const u32* __restrict__ pl_off,
                                                    const u32* __restrict__ pl_row, const double* __restrict__ pl_val,
                                                    const double* __restrict__ Z, int ldz, double* __restrict__ Y,
                                                    int ldy, const int* halt) {
    static_assert(NT == 32 || NT == SL_TB, "a warp or a CTA");
    if (halt && __ldcg(halt)) return;
    __shared__ __align__(16) double red[NT == 32 ? 1 : SL_TB / 32][4];
    const u32 Q = (u32(C) + 3) / 4, lane = threadIdx.x % NT;
    const size_t total = size_t(m) * Q, step = size_t(gridDim.x) * (SL_TB / NT);
    for (size_t q = (size_t(blockIdx.x) * SL_TB + threadIdx.x) / NT; q < total; q += step) {
        const u32 c = u32(q / Q);
        const int j = int(4 * (q % Q));
        V4<double> acc{0.0, 0.0, 0.0, 0.0};
        const u32 e1 = pl_off[c + 1];
#pragma unroll 4
        for (u32 e = pl_off[c] + lane; e < e1; e += NT) fma4(acc, pl_val[e], ld4(Z + size_t(pl_row[e]) * ldz + j));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            acc.a += __shfl_xor_sync(0xffffffffu, acc.a, o);
            acc.b += __shfl_xor_sync(0xffffffffu, acc.b, o);
            acc.c += __shfl_xor_sync(0xffffffffu, acc.c, o);
            acc.d += __shfl_xor_sync(0xffffffffu, acc.d, o);
        }
        double v = 0.0;  // lane k < 4 writes column j + k
        const u32 k = lane;
        if constexpr (NT == 32) {
            v = k == 0 ? acc.a : k == 1 ? acc.b : k == 2 ? acc.c : acc.d;
        } else {
            if (threadIdx.x % 32 == 0) st4s(red[threadIdx.x / 32], acc);
            __syncthreads();
            if (k < 4)
                for (int w = 0; w < SL_TB / 32; w++) v += red[w][k];
            __syncthreads();
        }
        if (k < 4 && j + int(k) < C) Y[size_t(c) * ldy + j + k] = v;
    }
}

// z = J r per block-Jacobi unit (b consecutive coordinates from c0, inverse at joff, b x b).
__global__ void __launch_bounds__(SL_TB) k_sl_jacobi(u32 nunits, int C, const u32* __restrict__ c0,
                                                      const u32* __restrict__ bw, const u32* __restrict__ joff,
                                                      const double* __restrict__ J, const double* __restrict__ r,
                                                      double* __restrict__ z, int ld) {
    const size_t total = size_t(nunits) * C;
    for (size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q < total; q += size_t(gridDim.x) * blockDim.x) {
        const u32 u = u32(q / C);
        const int j = int(q % C);
        const u32 b = bw[u], base = c0[u];
        const double* Ju = J + joff[u];
        double rr[SL_B_MAX];
#pragma unroll
        for (int a = 0; a < SL_B_MAX; a++) rr[a] = a < int(b) ? r[size_t(base + a) * ld + j] : 0.0;
        for (u32 a = 0; a < b; a++) {
            double v = 0.0;
#pragma unroll
            for (int bb = 0; bb < SL_B_MAX; bb++)
                if (bb < int(b)) v += Ju[a * b + bb] * rr[bb];
            z[size_t(base + a) * ld + j] = v;
        }
    }
}

}  // namespace fereg
