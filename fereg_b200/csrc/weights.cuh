// Device refresh of the weight state (operator.rs:211-338 refresh_weights, :344-570
// level_weights): cell weights W_c = sum of the cell's row weights, n1_s = sum of the segment's
// W_c, and for every reduced coordinate k: n_k = sum of W_c over the cells of k, and
// diag_k = n_k - sum_s c_{s,k}^2 / n1_s with c_{s,k} the weight of k's cells in segment s; k is
// redundant when diag_k <= 1e-12 n_k (operator.rs:21), and the Jacobi factor is 1 / diag_k
// otherwise. The coordinate-sorted lists hold each coordinate's cells in cell order, hence in
// segment order, so c_{s,k} are the sums over runs of equal segment: warps walk chunks of the
// lists 32 entries at a time with a segmented scan, and a per-coordinate pass stitches the runs
// that cross chunk boundaries. All sums have a fixed order.
#pragma once

#include "device.cuh"

namespace fereg {

// flag = 1 when a weight is not positive and finite.
__global__ void k_check_weights(const double* __restrict__ w, size_t n, int* flag) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const double x = w[i];
        if (!(x > 0.0 && x <= 1.7976931348623157e308)) atomicExch(flag, 1);
    }
}

// W_c = sum of the row weights of cell c (rows cell_row[c] .. cell_row[c+1]); flag (non-null): as
// k_check_weights.
__global__ void k_cell_weights(const double* __restrict__ w, const u32* __restrict__ cell_row, u32 M,
                               double* __restrict__ cw, int* __restrict__ flag) {
    for (u32 c = blockIdx.x * blockDim.x + threadIdx.x; c < M; c += gridDim.x * blockDim.x) {
        double s = 0.0;
        bool bad = false;
        for (u32 r = cell_row[c]; r < cell_row[c + 1]; r++) {
            const double x = w[r];
            bad |= !(x > 0.0 && x <= 1.7976931348623157e308);
            s += x;
        }
        if (flag && bad) atomicExch(flag, 1);
        cw[c] = s;
    }
}

// out[r] = in[pi[r]]: kept-order values in row order.
__global__ void k_gather_rows_f64(const double* __restrict__ in, const u32* __restrict__ pi, size_t n,
                                  double* __restrict__ out) {
    for (size_t r = size_t(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += size_t(gridDim.x) * blockDim.x)
        out[r] = in[pi[r]];
}

// pw[e] = the weight of list entry e's cell: the list passes of the operator then read the weights in
// order (4e6 entries, 4 columns: 67 -> 53 us an apply with the direct reads they allow
// (36 since the gathers are of 256 bits), 19 us per weight state).
__global__ void k_list_weights(const double* __restrict__ cw, const u32* __restrict__ pl_cell, size_t E,
                               double* __restrict__ pw) {
    for (size_t e = size_t(blockIdx.x) * blockDim.x + threadIdx.x; e < E; e += size_t(gridDim.x) * blockDim.x)
        pw[e] = cw[pl_cell[e]];
}

// W_c = the number of rows of cell c (unit row weights).
__global__ void k_cell_counts(const u32* __restrict__ cell_row, u32 M, double* __restrict__ cw) {
    for (u32 c = blockIdx.x * blockDim.x + threadIdx.x; c < M; c += gridDim.x * blockDim.x)
        cw[c] = double(cell_row[c + 1] - cell_row[c]);
}

// n1_s = sum of W_c over the segment's cells (cw null: 1 per cell); n1inv = 1 / n1.
__global__ void k_seg_weights(const double* __restrict__ cw, const u32* __restrict__ seg_off, u32 g1,
                              double* __restrict__ n1, double* __restrict__ n1inv) {
    for (u32 s = blockIdx.x * blockDim.x + threadIdx.x; s < g1; s += gridDim.x * blockDim.x) {
        double a = 0.0;
        for (u32 c = seg_off[s]; c < seg_off[s + 1]; c++) a += cw ? cw[c] : 1.0;
        n1[s] = a;
        n1inv[s] = 1.0 / a;
    }
}

// n_k, diag_k, redundant_k and the Jacobi factor of every coordinate, in two passes so that a
// long list (a 10-level year block holds n/10 entries per list) does not serialize on one warp.
//
// Pass 1, a warp per chunk of at most CW_CHUNK entries of one list: the chunk's sum of weights,
// its sum of squared runs as if the chunk were the whole list (dq_iso = sum_runs x^2 / n1_s), and
// its first and last runs (segment, partial sum). A segment's entries are contiguous in a list
// (lists are in cell order, cells in segment order), so the first run is every entry of the
// first entry's segment, and likewise for the last.
constexpr u32 CW_CHUNK = 512;

struct CwChunk {
    double nr, dq, xf, xl;
    u32 sf, sl;
};

__global__ void k_coord_chunks(const u32* __restrict__ chunk_e0, const u32* __restrict__ chunk_e1, u32 nchunks,
                               const u32* __restrict__ pl_cell, const u32* __restrict__ pl_seg,
                               const double* __restrict__ cw, const double* __restrict__ n1inv,
                               CwChunk* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const size_t gw = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5, nw = (size_t(gridDim.x) * blockDim.x) >> 5;
    constexpr u32 NONE = 0xffffffffu;
    for (size_t c = gw; c < nchunks; c += nw) {
        const u32 e0 = chunk_e0[c], e1 = chunk_e1[c];
        const u32 sf = pl_seg[e0], sl = pl_seg[e1 - 1];
        double nr_acc = 0.0, dq_acc = 0.0, xf = 0.0, xl = 0.0;
        u32 carry_s = NONE;
        double carry = 0.0;
        for (u32 base = e0; base < e1; base += 32) {
            const u32 e = base + u32(lane);
            const bool valid = e < e1;
            const double wv = valid ? (cw ? cw[pl_cell[e]] : 1.0) : 0.0;
            const u32 s = valid ? pl_seg[e] : NONE;
            nr_acc += wv;
            if (s == sf) xf += wv;
            if (s == sl) xl += wv;
            // the run carried from the previous sub-chunk ends here unless this one continues it
            const u32 s0 = __shfl_sync(FULL, s, 0);
            if (lane == 0 && carry_s != NONE && s0 != carry_s) dq_acc += carry * carry * n1inv[carry_s];
            // inclusive scan of wv over the lane's run (runs are contiguous)
            double x = wv;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const double y = __shfl_up_sync(FULL, x, d);
                const u32 sy = __shfl_up_sync(FULL, s, d);
                if (lane >= d && sy == s) x += y;
            }
            if (valid && s == carry_s) x += carry;  // the run left open by the previous sub-chunk
            const u32 s_next = __shfl_down_sync(FULL, s, 1);
            const bool tail = valid && (lane == 31 || s_next != s);
            const int last = int(min(31u, e1 - 1 - base));
            const u32 s_last = __shfl_sync(FULL, s, last);
            const double x_last = __shfl_sync(FULL, x, last);
            const bool final_sub = base + 32 >= e1;
            if (tail && (final_sub || s != s_last)) dq_acc += x * x * n1inv[s];
            carry_s = s_last;
            carry = x_last;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            nr_acc += __shfl_down_sync(FULL, nr_acc, d);
            dq_acc += __shfl_down_sync(FULL, dq_acc, d);
            xf += __shfl_down_sync(FULL, xf, d);
            xl += __shfl_down_sync(FULL, xl, d);
        }
        if (lane == 0) out[c] = CwChunk{nr_acc, dq_acc, xf, xl, sf, sl};
    }
}

// Pass 2, a thread per coordinate: the chunks of its list in order. Sums of nr and dq_iso; a run
// that spans chunks (its parts x_i) contributes (sum x_i)^2 - sum x_i^2 more. Then diag_k =
// n_k - dq_k, redundant when diag_k <= 1e-12 n_k (operator.rs:21), Jacobi factor 1 / diag_k.
__global__ void k_coord_combine(const u32* __restrict__ list_chunk_off, u32 m, const CwChunk* __restrict__ ch,
                                const double* __restrict__ n1inv, double* __restrict__ nr, double* __restrict__ diag,
                                uint8_t* __restrict__ red, double* __restrict__ inv_diag) {
    constexpr u32 NONE = 0xffffffffu;
    for (u32 k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        double n_acc = 0.0, dq = 0.0, X = 0.0, Q = 0.0, csn = 0.0;  // csn: 1 / n1 of segment cs
        u32 cs = NONE;
        const u32 cb = list_chunk_off[k], ce = list_chunk_off[k + 1];
        for (u32 c0 = cb; c0 < ce; c0 += 4) {
            CwChunk hh[4];  // four chunks' loads in flight (a list of 117 chunks took 83 us one by one)
            double ni[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (c0 + u < ce) hh[u] = ch[c0 + u];
#pragma unroll
            for (int u = 0; u < 4; u++) ni[u] = c0 + u < ce ? n1inv[hh[u].sf] : 0.0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (c0 + u >= ce) break;
                const CwChunk& h = hh[u];
                n_acc += h.nr;
                dq += h.dq;
                if (h.sf == cs) {
                    X += h.xf;
                    Q += h.xf * h.xf;
                } else {
                    if (cs != NONE) dq += (X * X - Q) * csn;
                    cs = h.sf;
                    csn = ni[u];
                    X = h.xf;
                    Q = h.xf * h.xf;
                }
                if (h.sl != h.sf) {  // the chunk holds more runs: the carried run ends at its first
                    dq += (X * X - Q) * csn;
                    cs = h.sl;
                    csn = n1inv[h.sl];
                    X = h.xl;
                    Q = h.xl * h.xl;
                }
            }
        }
        if (cs != NONE) dq += (X * X - Q) * csn;
        const double dg = n_acc - dq;
        const bool r = dg <= 1e-12 * n_acc;
        nr[k] = n_acc;
        diag[k] = dg;
        red[k] = r ? 1 : 0;
        inv_diag[k] = (r || !(dg > 0.0)) ? 0.0 : 1.0 / dg;
    }
}

// Dense small super-block S_SS (ms x ms, the first ms coordinates, ns small blocks) for the current
// cell weights (operator.rs:1457-1523, as the host assembly of the dense factor):
//   S_SS[k][l] = sum_c W_c [k in c][l in c] - sum_s c_{s,k} c_{s,l} / n1_s,
// c_{s,k} the weight of the cells of segment s that hold k. The first sum's diagonal is nr_k, the
// rest of it is nonzero between different small blocks only (k_small_cross). The second sum is a
// Gram matrix over the segments, formed as one (k_small_gram) where the segments times the tiles of
// the matrix do not pass the cells times ns, and by walking the few pairs that a segment's cells
// have (k_small_rows) beyond: a tile costs about 0.6 ns a segment, a cell's code about 1 ns. Measured
// with 10 cells a segment, both sums: 1e6 segments and 10 coordinates 0.16 ms (7.5 ms by lists, a
// lane at a time, before), 1e6 and 110 2.2 ms (20.0), 2e4 and 310 0.20 ms by tiles and 0.31 by
// lists, 2e5 and 910 4.2 ms by lists (6.4), where the 120 tiles would take 14; one unweighted block
// keeps the order it always had (k_small_ordered). Every sum has a fixed
// order.
//
// Partial row k of the first sum by work items (row k, a run of its list's entries): a warp takes
// 32 entries at a time, the lanes that meet in a code are added in lane order by the first of
// them, and that lane adds the sum to the item's row in shared memory. What bounds it is the
// latency of the gathers of the cells' codes, which some thousand items hide.
__device__ __forceinline__ void add_by_code(double* row, u32 code, double w, bool on, u32 lane) {
    const unsigned same = __match_any_sync(FULL, on ? code : 0x80000000u + lane);
    unsigned rest = same & ~((2u << lane) - 1u);  // the lanes after this one with its code
    if ((same & ((1u << lane) - 1u)) != 0) rest = 0;  // a lane before this one adds
    double sum = w;
    for (unsigned any = __ballot_sync(FULL, rest != 0); any; any = __ballot_sync(FULL, rest != 0)) {
        const int src = rest ? __ffs(int(rest)) - 1 : int(lane);
        const double v = __shfl_sync(FULL, w, src);
        if (rest) sum += v;
        rest &= rest - 1;
    }
    if (on && (same & ((1u << lane) - 1u)) == 0) row[code] += sum;
    __syncwarp();
}

__global__ void __launch_bounds__(256) k_small_cross(const u32* __restrict__ coord, u32 M, int ns, u32 ms,
                                                     const double* __restrict__ cw, const u32* __restrict__ pl_cell,
                                                     const u32* __restrict__ item_k, const u32* __restrict__ item_a,
                                                     const u32* __restrict__ item_b, u32 nitems,
                                                     double* __restrict__ part) {
    extern __shared__ double rows_s[];
    const u32 w = threadIdx.x / 32, lane = threadIdx.x % 32;
    const u32 it = blockIdx.x * 8 + w;
    if (it >= nitems) return;  // whole warps
    double* row = rows_s + size_t(w) * ms;
    for (u32 l = lane; l < ms; l += 32) row[l] = 0.0;
    __syncwarp();
    const u32 k = item_k[it], b = item_b[it];
    for (u32 base = item_a[it]; base < b; base += 32) {
        const u32 e = base + lane;
        const bool valid = e < b;
        const u32 c = valid ? pl_cell[e] : 0u;
        const double wc = valid ? (cw ? cw[c] : 1.0) : 0.0;
        for (int q = 0; q < ns; q++) {
            const u32 code = valid ? coord[size_t(q) * M + c] : k;
            add_by_code(row, code, wc, code != k, lane);  // the diagonal is nr_k
        }
    }
    for (u32 l = lane; l < ms; l += 32) part[size_t(it) * ms + l] = row[l];
}

// The same items when the second sum is added here too: for every segment of the run (an entry
// opens one where its segment differs from the list's entry before it), with c_{s,k} from the
// segment's cells, S[k][l] -= c_{s,k} W_c' / n1_s for the small codes l of every cell c' of s.
__global__ void __launch_bounds__(256) k_small_rows(const u32* __restrict__ seg_off, const u32* __restrict__ coord,
                                                    u32 M, int ns, u32 ms, const double* __restrict__ cw,
                                                    const double* __restrict__ n1inv, const u32* __restrict__ pl_off,
                                                    const u32* __restrict__ pl_cell, const u32* __restrict__ pl_seg,
                                                    const u32* __restrict__ item_k, const u32* __restrict__ item_a,
                                                    const u32* __restrict__ item_b, u32 nitems,
                                                    double* __restrict__ part) {
    extern __shared__ double rows_s[];
    const u32 w = threadIdx.x / 32, lane = threadIdx.x % 32;
    const u32 it = blockIdx.x * 8 + w;
    if (it >= nitems) return;  // whole warps
    double* row = rows_s + size_t(w) * ms;
    for (u32 l = lane; l < ms; l += 32) row[l] = 0.0;
    __syncwarp();
    const u32 k = item_k[it], b = item_b[it], first = pl_off[k];
    for (u32 base = item_a[it]; base < b; base += 32) {
        const u32 e = base + lane;
        const bool valid = e < b;
        const u32 c = valid ? pl_cell[e] : 0u, s = valid ? pl_seg[e] : 0u;
        const double wc = valid ? (cw ? cw[c] : 1.0) : 0.0;
        for (int q = 0; q < ns; q++) {
            const u32 code = valid ? coord[size_t(q) * M + c] : k;
            add_by_code(row, code, wc, code != k, lane);
        }
        const bool opens = valid && (e == first || pl_seg[e - 1] != s);
        const u32 c0 = opens ? seg_off[s] : 0u, c1 = opens ? seg_off[s + 1] : 0u;
        const double ni = opens ? n1inv[s] : 0.0;
        for (unsigned todo = __ballot_sync(FULL, opens); todo; todo &= todo - 1) {
            const int src = __ffs(int(todo)) - 1;
            const u32 a0 = __shfl_sync(FULL, c0, src), a1 = __shfl_sync(FULL, c1, src);
            double ck = 0.0;
            for (u32 cc = a0 + lane; cc < a1; cc += 32) {
                const double v = cw ? cw[cc] : 1.0;
                for (int q = 0; q < ns; q++)
                    if (coord[size_t(q) * M + cc] == k) ck += v;
            }
#pragma unroll
            for (int o = 16; o > 0; o /= 2) ck += __shfl_xor_sync(FULL, ck, o);
            const double f = ck * __shfl_sync(FULL, ni, src);
            for (u32 cb = a0; cb < a1; cb += 32) {
                const u32 cc = cb + lane;
                const bool on = cc < a1;
                const double v = on ? -f * (cw ? cw[cc] : 1.0) : 0.0;
                for (int q = 0; q < ns; q++) add_by_code(row, on ? coord[size_t(q) * M + cc] : 0u, v, on, lane);
            }
        }
    }
    for (u32 l = lane; l < ms; l += 32) part[size_t(it) * ms + l] = row[l];
}

// One unweighted small block of at most 32 coordinates, by the lists' entries in order: the partial
// row of an item (row k, a run of its list that never splits a segment), a lane per coordinate l.
// For every entry S[k][k] += 1; once per segment s of the run S[k][l] -= c_{s,k} / n1_s for each of the
// c_{s,l} cells that hold l (csk: the counts, g1 x ms). A lane's sum is one chain over the item, in
// entry order; the loads of 8 entries are in flight together. This is the block of a panel's years
// on a one-row-per-cell panel, whose order of sums is frozen as that of the vector steps is (pcg.cuh);
// blocks of every other shape take the faster forms above.
// 1e6 segments of 10 cells, 10 coordinates: 7.5 ms with one lane an item, 0.70 ms here (0.16 as tiles).
__global__ void __launch_bounds__(256) k_small_ordered(u32 ms, const double* __restrict__ n1inv,
                                                       const double* __restrict__ csk, const u32* __restrict__ pl_seg,
                                                       const u32* __restrict__ item_k, const u32* __restrict__ item_a,
                                                       const u32* __restrict__ item_b, u32 nitems,
                                                       double* __restrict__ part) {
    constexpr int U = 8;
    constexpr u32 NONE = 0xffffffffu;
    const u32 lane = threadIdx.x % 32;
    const u32 it = blockIdx.x * 8 + threadIdx.x / 32;
    if (it >= nitems) return;  // whole warps
    const u32 k = item_k[it], b = item_b[it];
    double acc = 0.0;
    u32 prev = NONE;
    for (u32 base = item_a[it]; base < b; base += 32) {
        const u32 e = base + lane;
        const u32 s = e < b ? pl_seg[e] : NONE;
        const double ni = e < b ? n1inv[s] : 0.0;
        const u32 left = __shfl_up_sync(FULL, s, 1);
        const bool opens = e < b && s != (lane == 0 ? prev : left);  // a segment's entries are consecutive
        const unsigned open = __ballot_sync(FULL, opens);
        const int n = int(min(32u, b - base));
        for (int j0 = 0; j0 < n; j0 += U) {
            double c[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const u32 sj = __shfl_sync(FULL, s, j0 + u);
                c[u] = (j0 + u < n && lane < ms) ? csk[size_t(sj) * ms + lane] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const double f = __shfl_sync(FULL, c[u], int(k)) * __shfl_sync(FULL, ni, j0 + u);
                if (j0 + u < n) {
                    if (lane == k) acc += 1.0;
                    if ((open >> (j0 + u)) & 1u)
                        for (int q = int(c[u]); q > 0; q--) acc -= f;
                }
            }
        }
        prev = __shfl_sync(FULL, s, n - 1);
    }
    if (lane < ms) part[size_t(it) * ms + lane] = acc;
}

// Row k of S_SS: the partial rows of k's items (first[k] .. first[k+1]) added in item order.
__global__ void k_small_items_sum(const double* __restrict__ part, const u32* __restrict__ first, u32 ms,
                                  double* __restrict__ out) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ms * ms) return;
    const u32 k = i / ms, l = i % ms;
    double v = 0.0;
#pragma unroll 16
    for (u32 it = first[k]; it < first[k + 1]; it++) v += part[size_t(it) * ms + l];
    out[i] = v;
}

// The Gram matrix sum_s c_s c_s' / n1_s by tiles of BT x BT (tile (ti, tj), tj <= ti, in blockIdx.y;
// blockIdx.x takes the segment chunks x, x + gridDim.x, ...): a chunk's rows c_s are summed into
// shared memory, thread (segment, small block) walking the segment's cells in order (a block's
// codes have their own columns, so no two threads share a slot), then every thread adds the
// products of its PT x PT outputs, segments in order. part[(y gridDim.x + x) BT BT + r BT + c].
template <int BT>
struct SgTile {
    static constexpr int TS = BT == 16 ? 64 : 32;   // segments per chunk
    static constexpr int PT = BT / 16;              // outputs per thread and side (16 x 16 threads)
    static constexpr int LD = BT + 1;
};
template <int BT>
__global__ void __launch_bounds__(256) k_small_gram(const u32* __restrict__ seg_off, const u32* __restrict__ coord,
                                                    u32 M, u32 g1, int ns, const double* __restrict__ cw,
                                                    const double* __restrict__ n1inv, double* __restrict__ part) {
    using T = SgTile<BT>;
    __shared__ double Ci[T::TS * T::LD], Cj[T::TS * T::LD], ni[T::TS];
    int ti = 0;
    while ((ti + 1) * (ti + 2) / 2 <= int(blockIdx.y)) ti++;
    const int tj = int(blockIdx.y) - ti * (ti + 1) / 2;
    const u32 ki = u32(ti * BT), kj = u32(tj * BT);
    const int tx = int(threadIdx.x % 16), ty = int(threadIdx.x / 16);
    double acc[T::PT][T::PT] = {};
    const double* B = ti == tj ? Ci : Cj;
    for (u32 s0 = blockIdx.x * T::TS; s0 < g1; s0 += gridDim.x * T::TS) {
        const u32 nseg = min(u32(T::TS), g1 - s0);
        __syncthreads();
        for (int i = threadIdx.x; i < T::TS * T::LD; i += 256) {
            Ci[i] = 0.0;
            if (ti != tj) Cj[i] = 0.0;
        }
        if (threadIdx.x < T::TS) ni[threadIdx.x] = threadIdx.x < nseg ? n1inv[s0 + threadIdx.x] : 0.0;
        __syncthreads();
        for (u32 i = threadIdx.x; i < nseg * u32(ns); i += 256) {
            const u32 sl = i % nseg, q = i / nseg;
            const u32* cd = coord + size_t(q) * M;
            const u32 c1 = seg_off[s0 + sl + 1];
#pragma unroll 4
            for (u32 c = seg_off[s0 + sl]; c < c1; c++) {
                const u32 code = cd[c];
                const double w = cw ? cw[c] : 1.0;
                if (code - ki < u32(BT)) Ci[sl * T::LD + (code - ki)] += w;
                if (ti != tj && code - kj < u32(BT)) Cj[sl * T::LD + (code - kj)] += w;
            }
        }
        __syncthreads();
        for (u32 sl = 0; sl < nseg; sl++) {
            double x[T::PT], y[T::PT];
            const double n = ni[sl];
#pragma unroll
            for (int r = 0; r < T::PT; r++) {
                x[r] = Ci[sl * T::LD + ty + 16 * r] * n;
                y[r] = B[sl * T::LD + tx + 16 * r];
            }
#pragma unroll
            for (int r = 0; r < T::PT; r++)
#pragma unroll
                for (int c = 0; c < T::PT; c++) acc[r][c] += x[r] * y[c];
        }
    }
    double* o = part + (size_t(blockIdx.y) * gridDim.x + blockIdx.x) * (BT * BT);
#pragma unroll
    for (int r = 0; r < T::PT; r++)
#pragma unroll
        for (int c = 0; c < T::PT; c++) o[(ty + 16 * r) * BT + tx + 16 * c] = acc[r][c];
}

// S_SS[k][l] from nr, the items' partial rows (row k: items first[k] .. first[k+1], in order; null:
// none) and, when gram is set, the tiles of k_small_gram (nsplit partials each): a warp per
// element of the lower triangle, lane i adding the partials i, i + 32, ... and a fixed butterfly;
// the upper triangle is its mirror.
template <int BT>
__global__ void k_small_combine(const double* __restrict__ items, const u32* __restrict__ first,
                                const double* __restrict__ gram, u32 nsplit, const double* __restrict__ nr, u32 ms,
                                double* __restrict__ out) {
    const u32 lane = threadIdx.x & 31u;
    const size_t gw = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5, nw = (size_t(gridDim.x) * blockDim.x) >> 5;
    for (size_t e = gw; e < size_t(ms) * ms; e += nw) {
        const u32 k = u32(e / ms), l = u32(e % ms);
        if (l > k) continue;
        double v = 0.0, g = 0.0;
        if (items)
            for (u32 it = first[k] + lane; it < first[k + 1]; it += 32) v += items[size_t(it) * ms + l];
        if (gram) {
            const u32 ti = k / BT, tj = l / BT;
            const double* t = gram + size_t(ti * (ti + 1) / 2 + tj) * nsplit * (BT * BT) + (k % BT) * BT + l % BT;
            for (u32 x = lane; x < nsplit; x += 32) g += t[size_t(x) * (BT * BT)];
        }
        v -= g;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if (k == l) v += nr[k];
        if (lane == 0) out[size_t(k) * ms + l] = out[size_t(l) * ms + k] = v;
    }
}

// ak (k x k) = the kept rows / columns of a (ms x ms), scaled to unit diagonal.
__global__ void k_small_gather(const double* __restrict__ a, u32 ms, const u32* __restrict__ keep,
                               const double* __restrict__ scale, int k, double* __restrict__ ak) {
    const size_t total = size_t(k) * k;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
        const int r = int(i / k), c = int(i % k);
        ak[i] = a[size_t(keep[r]) * ms + keep[c]] * scale[r] * scale[c];
    }
}

// Sum of a vector into per-CTA partials (fixed tree); the host adds the partials in CTA order.
__global__ void __launch_bounds__(256) k_vec_sum(const double* __restrict__ v, size_t n, double* __restrict__ part) {
    __shared__ double red[256];
    double s = 0.0;
    for (size_t i = size_t(blockIdx.x) * 256 + threadIdx.x; i < n; i += size_t(gridDim.x) * 256) s += v[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// ---------------------------------------------------------------------------------------------
// The rows of S on the small coordinates, for the operator (operator.rs:894-948 restated as a
// product): with at most SACC_MAX small coordinates (blocks 0..ns-1, coordinates 0..ms-1),
//   S[k][f] = sum_{c containing k and f} W_c - sum_s c_{s,k} c_{s,f} / n1_s,
// with c_{s,k} the weight of the cells of segment s that hold k. The operator then takes
// Y[k] = sum_f S[k][f] P[f] for the small k from this dense ms x m block (stored transposed,
// srow[f * ms + k], f over every coordinate) instead of accumulating per cell in the segment
// pass. srow depends on the weights: it is rebuilt with every weight state.

// c_{s,k} for every segment s and small coordinate k < ms: one thread per (segment, k), the
// segment's cells in order.
__global__ void k_seg_small_w(const u32* __restrict__ seg_off, const u32* __restrict__ coord, u32 M, u32 g1, int ns,
                              u32 ms, const double* __restrict__ cw, double* __restrict__ csk) {
    const size_t total = size_t(g1) * ms;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
        const u32 s = u32(i / ms), k = u32(i % ms);
        double a = 0.0;
        for (u32 c = seg_off[s]; c < seg_off[s + 1]; c++) {
            const double w = cw ? cw[c] : 1.0;
            for (int b = 0; b < ns; b++)
                if (coord[size_t(b) * M + c] == k) a += w;
        }
        csk[i] = a;
    }
}

// Partial rows of srow by work items: item i covers entries [item_a, item_b) of the coordinate
// list of f = item_f (whole runs of equal segment). One warp per item, lane k < ms holding
// S[k][f] over the item: for every entry (cell c of segment s) W_c when c holds k; at the end of
// each run of segment s, - c_{s,k} c_{s,f} / n1_s with c_{s,f} the run's weight sum. Every lane
// sums in entry order; k_srow_sum adds the items of a coordinate in item order.
__global__ void __launch_bounds__(256) k_srow_items(const u32* __restrict__ coord, u32 M, int ns, u32 ms,
                                                    const double* __restrict__ cw, const double* __restrict__ n1inv,
                                                    const u32* __restrict__ pl_cell, const u32* __restrict__ pl_seg,
                                                    const double* __restrict__ csk, const u32* __restrict__ item_a,
                                                    const u32* __restrict__ item_b, u32 nitems,
                                                    double* __restrict__ part) {
    const u32 lane = threadIdx.x & 31u;
    const u32 it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (it >= nitems) return;  // whole warps
    const u32 b = item_b[it];
    double acc = 0.0, run = 0.0;
    for (u32 e = item_a[it]; e < b; e++) {
        const u32 c = pl_cell[e], s = pl_seg[e];
        const double w = cw ? cw[c] : 1.0;
        for (int bb = 0; bb < ns; bb++)
            if (coord[size_t(bb) * M + c] == lane) acc += w;
        run += w;
        if (e + 1 == b || pl_seg[e + 1] != s) {
            if (lane < ms) acc -= csk[size_t(s) * ms + lane] * run * n1inv[s];
            run = 0.0;
        }
    }
    if (lane < ms) part[size_t(it) * ms + lane] = acc;
}

// srow[f * ms + k] = the partial rows of f's items (first[f] .. first[f+1]) added in item order.
__global__ void k_srow_sum(const double* __restrict__ part, const u32* __restrict__ first, u32 m, u32 ms,
                           double* __restrict__ srow) {
    const size_t total = size_t(m) * ms;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
        const u32 f = u32(i / ms), k = u32(i % ms);
        double v = 0.0;
        for (u32 it = first[f]; it < first[f + 1]; it++) v += part[size_t(it) * ms + k];
        srow[i] = v;
    }
}

// Exact leverage of the fixed-effect columns per row (leverage.rs:128 fe_hat, by block
// elimination of FE1): h_i = w_i (1 / W_s + v_c' G v_c) for row i of cell c in segment s, where
// v_c = b_c - t_s, b_c the indicator of c's reduced coordinates, t_s = sum_{c' in s} W_c' b_c' / W_s
// and G a generalized inverse of the reduced system S (any one: v_c lies in the range of
// S = sum_c W_c v_c v_c'). G: the dense m x m inverse. One thread per segment, cells in order.
__global__ void k_fe_leverage(DevStruct S, DevWeights W, const double* __restrict__ G, double* __restrict__ h) {
    const u32 m = S.m, M = S.M;
    for (u32 s = blockIdx.x * blockDim.x + threadIdx.x; s < S.g1; s += gridDim.x * blockDim.x) {
        const u32 c0 = S.seg_off[s], c1 = S.seg_off[s + 1];
        const double winv = W.n1inv[s];
        // B(c, c') = b_c' G b_c'
        auto B = [&](u32 c, u32 c2) {
            double v = 0.0;
            for (u32 k = 0; k < S.nb; k++)
                for (u32 l = 0; l < S.nb; l++)
                    v += G[size_t(S.coord[size_t(k) * M + c]) * m + S.coord[size_t(l) * M + c2]];
            return v;
        };
        double tau = 0.0;  // t' G t
        for (u32 c = c0; c < c1; c++) {
            double row = 0.0;
            for (u32 c2 = c0; c2 < c1; c2++) row += cellw(W, c2) * B(c, c2);
            tau += cellw(W, c) * row;
        }
        tau *= winv * winv;
        for (u32 c = c0; c < c1; c++) {
            double gt = 0.0;  // b_c' G t
            for (u32 c2 = c0; c2 < c1; c2++) gt += cellw(W, c2) * B(c, c2);
            const double q = m ? B(c, c) - 2.0 * gt * winv + tau : 0.0;
            for (u32 i = row0_of(S, c); i < row1_of(S, c); i++) h[i] = (W.w_rows ? W.w_rows[i] : 1.0) * (winv + q);
        }
    }
}

}  // namespace fereg
