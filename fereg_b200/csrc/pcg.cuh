// The PCG iteration's vector steps (cg.rs:132-292), each reducing its column sums in the same
// launch: every CTA writes its partials, and the CTA that finishes last (a ticket counter, after a
// memory fence) adds them in CTA order and applies the iteration's scalar step. Results are
// independent of which CTA finishes last.
//
// Up to WIDE_R columns (k_pq_gamma, k_update_xr, k_rz_stop) the vectors mostly sit in L2 and the
// chain of a step (loads, barrier, fence, ticket, the last CTA's partials and scalars) bounds it:
// the loads of a thread, of the partials and of the columns' state are in flight together, the
// preconditioner's Jacobi part is formed where r is. Their order of sums is frozen to a grid of
// VEC_GRID CTAs, whatever the size, for one shape's sake: unweighted cells of one row with one small
// block (a panel and its years). On a connected ring of firms the PCG of that shape ends at the
// round-off of these sums, and any other order moves the answer in its eighth digit. Systems whose
// order is not frozen take the wide steps where those are faster (weighted ones: 30 us an iteration
// for 43).
// Wider (a bootstrap's 512 columns: k_wide_*), the bytes bound the steps: CTA (x, y) takes rows of
// column tile y (VT columns), its threads are (row slot, quad of columns), so a row is read by
// neighbouring lanes in 32-byte pieces with VU rows in flight a thread, the small coordinates' rows
// of q = S p are formed beside p'q, and r'z, the small preconditioner and the stopping rule beside
// the update of r. 512 columns x 2e4 coordinates, an iteration's vector kernels: 560 -> 260 us.
//
// The iteration counter lives on the device, so the same kernels run launched one by one or as
// the body of a captured CUDA graph whose WHILE node repeats them. Each turn of the WHILE node costs
// 19 us between its body's last kernel and its first (0.2 us between two kernels of a body), so a
// body holds several iterations: k_update_p ends each by setting the next one's halt word (no column
// active, or the launch's cap of iterations reached), at which the kernels of the iterations behind
// it return at once, and the last one sets the loop condition. The counter rises with every iteration run, so
// a graph launch ends after at most `cap` iterations whatever the stopping rule does.
#pragma once

#include "kernels.cuh"

namespace fereg {

constexpr int WIDE_R = 64;  // the widest block of the narrow kernels
constexpr int VT = 64;      // columns per tile of the wide kernels
constexpr int VU = 4;       // rows in flight per thread
constexpr int VEC_GRID = 148 * 2;  // CTAs of the narrow kernels: the order of their sums

__host__ __device__ inline int vec_tiles(int R) { return (R + VT - 1) / VT; }
// CTAs per column tile: VU rows a thread, at most two CTAs an SM in all.
inline int vec_splits(u32 m, int R, int per_row) {
    const int Rc = R < VT ? R : VT, slots = TB / (Rc / 4 * per_row);
    const long long want = ((long long)m + (long long)slots * VU - 1) / ((long long)slots * VU);
    const int most = 296 / vec_tiles(R);
    return int(want < 1 ? 1 : want > (most > 1 ? most : 1) ? (most > 1 ? most : 1) : want);
}

// Device state of the iteration loop.
struct CgLoop {
    int* ctl;             // [n_active (mirrors CgState::n_active), k since the (re)start, k of this launch, cap, two halt words]
    const int* halt;      // this iteration's halt word: its kernels return when it is set
    int* halt_next;       // the next one's, set by k_update_p (null: no further iteration in the batch)
    const double* tol;    // the stopping rule's tolerance (set per solve, so that one graph serves every tolerance)
    unsigned* ticket;     // last-CTA counters: VTICKETS per kernel and column tile, then the finished tiles and their active columns
    double* rho_from;     // rho after iteration PROBE_FROM (cg.rs:24-37 probe)
    double* rho_at;       // rho after iteration PROBE_AT
    int* act_at;          // the column states after iteration PROBE_AT
    // The state as iteration u of a batch sees it; more: iteration u + 1 follows in the batch. (A
    // graph's body holds an even number of iterations, or one.)
    CgLoop at(int u, bool more) const {
        CgLoop l = *this;
        l.halt = ctl + 4 + (u & 1);
        l.halt_next = more ? ctl + 4 + ((u + 1) & 1) : nullptr;
        return l;
    }
};

// True in the CTA that is the last of `count` to get here; its loads of the others' results must
// bypass L1. The counter returns to 0.
__device__ __forceinline__ bool last_of(unsigned* ticket, unsigned count) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(ticket, 1u) == count - 1;
        if (last) *ticket = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// The calling thread's place in column tile blockIdx.y: quad q of row slot `slot` (per_row groups
// of quads share a row slot, `part` is the thread's among them).
struct VPlace {
    int c0, Rc, Q, nslot, slot, part, q;
    bool on;
    __device__ __forceinline__ VPlace(int R, int per_row) {
        c0 = int(blockIdx.y) * VT;
        Rc = min(VT, R - c0);
        Q = Rc / 4;
        const int w = Q * per_row;
        nslot = TB / w;
        slot = int(threadIdx.x) / w;
        part = int(threadIdx.x) % w / Q;
        q = int(threadIdx.x) % Q;
        on = slot < nslot;
    }
};

// out(o, sum over i < count of at(i, o)) for o < width (at most TB): the threads of group g add
// i = g, g + G, ... in order, thread o the groups' sums in order. Called by the whole CTA; `red`
// holds TB values and is free on return.
template <class T, class At, class Out>
__device__ __forceinline__ void grouped_sums(int count, int width, T* red, At&& at, Out&& out) {
    const int G = min(TB / width, count > 1 ? count : 1);
    const int o = int(threadIdx.x) % width, g = int(threadIdx.x) / width;
    T s = T(0);
    if (g < G) {
#pragma unroll 16
        for (int i = g; i < count; i += G) s += at(i, o);
    }
    if (G == 1) {
        if (g < 1) out(o, s);
    } else {
        if (g < G) red[g * width + o] = s;
        __syncthreads();
        if (int(threadIdx.x) < width) {
            T t = T(0);
            for (int i = 0; i < G; i++) t += red[i * width + o];
            out(o, t);
        }
    }
    __syncthreads();
}

// The sums over the CTAs of a column tile of their W partials each (part[x * stride + o], the tile's
// base in part): true in one CTA per tile, with the totals in fin. Past VGROUP CTAs in two stages,
// the last CTA of each VGROUP adding its group into the group's first slot: one CTA adding 296 rows
// of 156 partials takes longer than the product itself. tk: 1 + the groups' counters.
constexpr int VGROUP = 24;
constexpr int VTICKETS = 1 + (296 + VGROUP - 1) / VGROUP;  // counters per tile and kernel
__device__ __forceinline__ bool tile_sums(double* part, int W, size_t stride, unsigned* tk, double* red2, double* fin) {
    int n = int(gridDim.x);
    size_t st = stride;
    if (n > VGROUP) {
        const int grp = int(blockIdx.x) / VGROUP, gs = min(VGROUP, n - grp * VGROUP);
        if (!last_of(tk + 1 + grp, unsigned(gs))) return false;
        double* base = part + size_t(grp) * VGROUP * stride;
        for (int o0 = 0; o0 < W; o0 += TB)
            grouped_sums(gs, min(TB, W - o0), red2, [&](int i, int o) { return __ldcg(base + size_t(i) * stride + o0 + o); },
                         [&](int o, double t) { base[o0 + o] = t; });
        n = (n + VGROUP - 1) / VGROUP;
        st = size_t(VGROUP) * stride;
    }
    if (!last_of(tk, unsigned(n))) return false;
    for (int o0 = 0; o0 < W; o0 += TB)
        grouped_sums(n, min(TB, W - o0), red2, [&](int i, int o) { return __ldcg(part + size_t(i) * st + o0 + o); },
                     [&](int o, double t) { fin[o0 + o] = t; });
    return true;
}

__device__ __forceinline__ V4<double> ldv(const double* p) {
    V4<double> v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.a), "=d"(v.b), "=d"(v.c), "=d"(v.d) : "l"(p));
    return v;
}
__device__ __forceinline__ V4<float> ldv(const float* p) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    return V4<float>{x.x, x.y, x.z, x.w};
}
template <class T>
__device__ __forceinline__ void dot4(V4<double>& s, const V4<T>& a, const V4<T>& b) {
    s.a += double(a.a) * double(b.a);
    s.b += double(a.b) * double(b.b);
    s.c += double(a.c) * double(b.c);
    s.d += double(a.d) * double(b.d);
}
template <class T>
__device__ __forceinline__ void put4(T* red, const V4<T>& v) {
    red[0] = v.a;
    red[1] = v.b;
    red[2] = v.c;
    red[3] = v.d;
}

// The active columns' count of the tiles that have finished; the last tile publishes it and the
// iteration number. Called by one thread per tile.
__device__ __forceinline__ void tile_done(const CgState& st, const CgLoop& lp, int k, unsigned active) {
    unsigned* done = lp.ticket + 3 * VTICKETS * gridDim.y;
    atomicAdd(done + 1, active);  // integer counts: order independent
    __threadfence();
    if (atomicAdd(done, 1u) == gridDim.y - 1) {
        __threadfence();
        const int n = int(atomicExch(done + 1, 0u));
        *done = 0;
        *st.n_active = n;
        lp.ctl[0] = n;
        lp.ctl[1] = k;
    }
}

// A column's state as the stopping rule reads it, loaded before the sums arrive (one after another
// behind them the loads cost as much as the sums).
struct ColState {
    double ring[WINDOW], gamma, rho, ss1, xconst, floor_, pfloor, tol;
    int active, k;
    __device__ __forceinline__ void load(const CgState& st, const CgLoop& lp, int j) {
#pragma unroll
        for (int w = 0; w < WINDOW; w++) ring[w] = st.ring[size_t(j) * WINDOW + w];
        gamma = st.gamma[j];
        rho = st.rho[j];
        ss1 = st.ss1[j];
        xconst = st.xconst[j];
        floor_ = st.floor_[j];
        pfloor = st.pfloor[j];
        tol = *lp.tol;
        active = st.active[j];
        k = lp.ctl[1] + 1;
    }
};

// The stopping rule (cg.rs:239-253) and beta of column j, given rho_new = r'z and
// xsum = x0'rhs + x'rhs + x'r + x0'r; the probe's contraction inputs are recorded at probe_from and probe_at.
// Returns whether the column stays active.
__device__ __forceinline__ bool stop_column(const CgState& st, const CgLoop& lp, int j, ColState& c, double rn,
                                            double xsum, int probe_from, int probe_at) {
    double beta = 0.0;
    const int k = c.k;
    if (c.active == 1) {
        const double gr = c.gamma * c.rho;
        st.ring[size_t(j) * WINDOW + (k - 1) % WINDOW] = gr;
        const double ssk = c.ss1 - xsum;
        const double thr = fmax(c.tol * c.tol * ssk, c.floor_);
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < WINDOW; w++) sum += w == (k - 1) % WINDOW ? gr : c.ring[w];
        const bool done = k >= WINDOW && sum <= thr;
        const bool at_roundoff = rn <= c.floor_;
        // In an FP32 round (pfloor > 0) a breakdown or the FP32 round-off floor ends the round
        // with another FP64 restart (state 2); only the window rule stops the column.
        if (done) c.active = 0;
        else if (at_roundoff || !(rn > 0.0)) c.active = c.pfloor > 0.0 ? 2 : 0;
        else if (rn <= c.pfloor) c.active = 2;
        else beta = rn / c.rho;
        st.active[j] = c.active;
    }
    st.beta[j] = beta;
    st.rho[j] = rn;
    if (k == probe_from) lp.rho_from[j] = rn;
    if (k == probe_at) {
        lp.rho_at[j] = rn;
        lp.act_at[j] = c.active;
    }
    return c.active == 1;
}

// q[k] = sum_f S[k][f] p[f] for the small k < ms from the dense rows of S (srow, weights.cuh; the
// caller wrote the other rows of q), then, with DOT, p'q and gamma = rho / p'q on the active columns
// (a non-positive or non-finite p'q deactivates). KQ = ceil(ms / 4) groups of quads share a row
// slot, group h holding the coordinates 4h .. 4h + 3; the first one forms the product p'q of the
// rows past ms. part: per CTA (4 KQ + 1) x Rc values of T and double (double storage).
template <class T, int KQ, bool DOT>
__global__ void __launch_bounds__(TB) k_wide_pq(const double* __restrict__ srow, u32 ms, const T* __restrict__ p,
                                                 T* __restrict__ q, u32 m, int R, double* __restrict__ part, CgState st,
                                                 CgLoop lp) {
    constexpr int PR = KQ > 0 ? KQ : 1;
    constexpr int NS = KQ > 0 ? 16 : 0;  // values of the small rows per thread
    __shared__ double red[TB * (NS + 4)], red2[TB];
    if (DOT && __ldcg(lp.halt)) return;
    double* fin = red;  // free once the CTA's own sums are out
    const VPlace v(R, PR);
    const u32 step = gridDim.x * u32(v.nslot);
    const size_t Ru = size_t(R);
    V4<T> acc[4] = {};
    V4<double> pq{0.0, 0.0, 0.0, 0.0};
    const int wk = 4 * KQ * v.Rc, W = wk + (DOT ? v.Rc : 0);  // sums per CTA
    if (v.on) {
        const T* pj = p + v.c0 + 4 * v.q;
        const T* qj = q + v.c0 + 4 * v.q;
        const u32 h = 4 * u32(v.part);
#pragma unroll VU
        for (u32 f = blockIdx.x * u32(v.nslot) + u32(v.slot); f < m; f += step) {
            const V4<T> x = ld4(pj + size_t(f) * Ru);
            if (DOT && v.part == 0 && f >= ms) dot4(pq, x, ldv(qj + size_t(f) * Ru));
            if constexpr (KQ > 0) {
                const double* sr = srow + size_t(f) * ms + h;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (h + k < ms) fma4(acc[k], T(__ldg(sr + k)), x);
            }
        }
        if constexpr (KQ > 0) {
            T* rt = reinterpret_cast<T*>(red) + size_t(v.slot) * wk + 4 * v.part * v.Rc + 4 * v.q;
#pragma unroll
            for (int k = 0; k < 4; k++) put4(rt + k * v.Rc, acc[k]);
        }
        if (DOT && v.part == 0) put4(red + TB * NS + v.slot * v.Rc + 4 * v.q, pq);
    }
    __syncthreads();
    const size_t stride = size_t((KQ * 4 + 1) * VT);
    double* tile = part + size_t(blockIdx.y) * gridDim.x * stride;
    double* mine = tile + size_t(blockIdx.x) * stride;
    if constexpr (KQ > 0) {
        const T* rt = reinterpret_cast<const T*>(red);
        for (int o0 = 0; o0 < wk; o0 += TB)
            grouped_sums(v.nslot, min(TB, wk - o0), reinterpret_cast<T*>(red2),
                         [&](int i, int o) { return rt[i * wk + o0 + o]; },
                         [&](int o, T s) { mine[o0 + o] = double(s); });
    }
    if constexpr (DOT)
        grouped_sums(v.nslot, v.Rc, red2, [&](int i, int o) { return red[TB * NS + i * v.Rc + o]; },
                     [&](int o, double s) { mine[wk + o] = s; });
    const int c = int(threadIdx.x), j = v.c0 + c;
    double rho = 0.0, pfl = 0.0;
    int act = 0;
    if (DOT && c < v.Rc) {
        rho = st.rho[j];
        pfl = st.pfloor[j];
        act = st.active[j];
    }
    if (!tile_sums(tile, W, stride, lp.ticket + VTICKETS * blockIdx.y, red2, fin)) return;
    // the small rows of q, and their share of p'q
    if constexpr (KQ > 0)
        for (int i = threadIdx.x; i < int(ms) * v.Rc; i += TB) {
            const int k = i / v.Rc, cc = i % v.Rc;
            const T y = T(fin[i]);
            q[size_t(k) * Ru + v.c0 + cc] = y;
            if (DOT) fin[i] = double(p[size_t(k) * Ru + v.c0 + cc]) * double(y);
        }
    if constexpr (DOT) {
        __syncthreads();
        if (c < v.Rc) {
            double s = fin[wk + c];
            if constexpr (KQ > 0)
                for (u32 k = 0; k < ms; k++) s += fin[int(k) * v.Rc + c];
            double g = 0.0;
            if (act == 1) {
                if (s > 0.0 && isfinite(s)) g = rho / s;
                else st.active[j] = pfl > 0.0 ? 2 : 0;  // inner rounds: FP64 restart, not a stop
            }
            st.gamma[j] = g;
        }
    }
}

// The largest small block (ms) whose product the last CTA of k_wide_xr forms itself: its rows of r
// for a column tile fit the staging buffer and the product stays at a few us for one SM.
constexpr int PRE_STAGE = 4096;
inline bool pre_fused(u32 ms, int R) {
    const u32 Rc = u32(R < VT ? R : VT);
    return ms * Rc <= u32(PRE_STAGE) && size_t(ms) * ms * Rc <= (size_t(1) << 17);
}

// x += gamma p, r -= gamma q, and the sums x'rhs, x'r, x0'r (x0 null: 0). PRE: also z = inv_diag r on
// the rows from ms on, z = minv r on the small ones (by the last CTA of each tile), r'z, the
// stopping rule and beta; otherwise the sums go to st.xb.
template <class T, bool PRE>
__global__ void __launch_bounds__(TB) k_wide_xr(T* __restrict__ x, T* __restrict__ r, const T* __restrict__ p,
                                                  const T* __restrict__ q, const T* __restrict__ rhs,
                                                  const T* __restrict__ x0, u32 m, int R, double* __restrict__ part,
                                                  CgState st, CgLoop lp, T* __restrict__ z,
                                                  const double* __restrict__ inv_diag, const double* __restrict__ minv,
                                                  u32 ms, int probe_from, int probe_at) {
    constexpr int NV = PRE ? 4 : 3;
    __shared__ double red[PRE_STAGE], red2[TB];
    __shared__ double fin[4 * VT];
    if (__ldcg(lp.halt)) return;
    const VPlace v(R, 1);
    const u32 step = gridDim.x * u32(v.nslot);
    const size_t Ru = size_t(R);
    V4<double> s[4] = {};
    if (v.on) {
        const int c = v.c0 + 4 * v.q;
        const T g0 = T(st.gamma[c]), g1 = T(st.gamma[c + 1]), g2 = T(st.gamma[c + 2]), g3 = T(st.gamma[c + 3]);
#pragma unroll 2
        for (u32 i = blockIdx.x * u32(v.nslot) + u32(v.slot); i < m; i += step) {
            const size_t o = size_t(i) * Ru + c;
            V4<T> xv = ldv(x + o), rv = ldv(r + o);
            const V4<T> pv = ld4(p + o), qv = ld4(q + o), bv = ld4(rhs + o);
            xv.a = xv.a + g0 * pv.a;
            xv.b = xv.b + g1 * pv.b;
            xv.c = xv.c + g2 * pv.c;
            xv.d = xv.d + g3 * pv.d;
            rv.a = rv.a - g0 * qv.a;
            rv.b = rv.b - g1 * qv.b;
            rv.c = rv.c - g2 * qv.c;
            rv.d = rv.d - g3 * qv.d;
            st4(x + o, xv);
            st4(r + o, rv);
            dot4(s[0], xv, bv);
            dot4(s[1], xv, rv);
            if (x0) dot4(s[2], ld4(x0 + o), rv);
            if constexpr (PRE)
                if (i >= ms) {
                    const T w = T(__ldg(inv_diag + i));
                    const V4<T> zv{w * rv.a, w * rv.b, w * rv.c, w * rv.d};
                    st4(z + o, zv);
                    dot4(s[3], rv, zv);
                }
        }
    }
    double* tile = part + size_t(blockIdx.y) * gridDim.x * size_t(NV * VT);
    double* mine = tile + size_t(blockIdx.x) * size_t(NV * VT);
    const int W = NV * v.Rc;
    if (v.on) {
#pragma unroll
        for (int k = 0; k < NV; k++) put4(red + v.slot * W + k * v.Rc + 4 * v.q, s[k]);
    }
    __syncthreads();
    grouped_sums(v.nslot, W, red2, [&](int i, int o) { return red[i * W + o]; }, [&](int o, double t) { mine[o] = t; });
    const int c = int(threadIdx.x), j = v.c0 + c;
    ColState cs;
    if (PRE && c < v.Rc) cs.load(st, lp, j);
    if (!tile_sums(tile, W, size_t(NV * VT), lp.ticket + VTICKETS * (gridDim.y + blockIdx.y), red2, fin)) return;
    if constexpr (!PRE) {
        if (c < v.Rc)
            for (int k = 0; k < 3; k++) st.xb[k * R + j] = fin[k * v.Rc + c];
        return;
    } else {
        double rz = c < v.Rc ? fin[3 * v.Rc + c] : 0.0;
        if (ms > 0) {
            for (int i = threadIdx.x; i < int(ms) * v.Rc; i += TB)
                red[i] = double(__ldcg(r + size_t(i / v.Rc) * Ru + v.c0 + i % v.Rc));
            __syncthreads();
            const int G = TB / v.Rc, o = int(threadIdx.x) % v.Rc, g = int(threadIdx.x) / v.Rc;
            double a = 0.0;
            if (g < G)
                for (u32 i = u32(g); i < ms; i += u32(G)) {
                    const double* mr = minv + size_t(i) * ms;
                    double zi = 0.0;
#pragma unroll 8
                    for (u32 l = 0; l < ms; l++) zi += __ldg(mr + l) * red[l * u32(v.Rc) + o];
                    const T zt = T(zi);
                    z[size_t(i) * Ru + v.c0 + o] = zt;
                    a += red[i * u32(v.Rc) + o] * double(zt);
                }
            if (g < G) red2[threadIdx.x] = a;
            __syncthreads();
            if (c < v.Rc)
                for (int i = 0; i < G; i++) rz += red2[i * v.Rc + c];
        }
        const bool live = c < v.Rc && stop_column(st, lp, j, cs, rz, cs.xconst + fin[c] + fin[v.Rc + c] + fin[2 * v.Rc + c],
                                                  probe_from, probe_at);
        const int n = __syncthreads_count(live);
        if (threadIdx.x == 0) tile_done(st, lp, cs.k, unsigned(n));
    }
}

// rho_new = r'z of a preconditioner applied by kernels of its own, then the stopping rule and
// beta. START: the rho of a (re)start instead (cg.rs:201-205): columns with rho <= 0 stop, the
// precision floor is drop rho, the active columns are counted.
template <class T, bool START>
__global__ void __launch_bounds__(TB) k_wide_rz(const T* __restrict__ r, const T* __restrict__ z, u32 m, int R,
                                                double* __restrict__ part, CgState st, CgLoop lp, int probe_from,
                                                int probe_at, double drop) {
    __shared__ double red[TB * 4], red2[TB];
    __shared__ double fin[VT];
    if (!START && __ldcg(lp.halt)) return;
    const VPlace v(R, 1);
    const u32 step = gridDim.x * u32(v.nslot);
    V4<double> s{0.0, 0.0, 0.0, 0.0};
    if (v.on) {
        const size_t c = size_t(v.c0 + 4 * v.q);
#pragma unroll VU
        for (u32 i = blockIdx.x * u32(v.nslot) + u32(v.slot); i < m; i += step)
            dot4(s, ld4(r + size_t(i) * R + c), ld4(z + size_t(i) * R + c));
        put4(red + v.slot * v.Rc + 4 * v.q, s);
    }
    __syncthreads();
    double* tile = part + size_t(blockIdx.y) * gridDim.x * size_t(VT);
    double* mine = tile + size_t(blockIdx.x) * size_t(VT);
    grouped_sums(v.nslot, v.Rc, red2, [&](int i, int o) { return red[i * v.Rc + o]; },
                 [&](int o, double t) { mine[o] = t; });
    const int c = int(threadIdx.x), j = v.c0 + c;
    ColState cs;
    double xsum = 0.0;
    if (!START && c < v.Rc) {
        cs.load(st, lp, j);
        xsum = cs.xconst + st.xb[j] + st.xb[R + j] + st.xb[2 * R + j];
    }
    if (!tile_sums(tile, v.Rc, size_t(VT), lp.ticket + VTICKETS * (2 * gridDim.y + blockIdx.y), red2, fin)) return;
    bool live = false;
    if (c < v.Rc) {
        if (START) {
            st.rho[j] = fin[c];
            if (st.active[j] == 1 && !(fin[c] > 0.0)) st.active[j] = 0;
            st.pfloor[j] = drop * fin[c];
            live = st.active[j] == 1;
        } else {
            live = stop_column(st, lp, j, cs, fin[c], xsum, probe_from, probe_at);
        }
    }
    const int n = __syncthreads_count(live);
    if (threadIdx.x == 0) tile_done(st, lp, START ? 0 : cs.k, unsigned(n));
}

// ---------------------------------------------------------------------------------------------
// Up to WIDE_R columns, on VEC_GRID CTAs. A CTA's partial of a column is the sum over its row slots
// (in order) of a thread's sum over the slot's rows (in order); the last CTA adds a column's partials
// with one warp, lane l the partials l, l + 32, ... in order, then a fixed butterfly.

// Sums of the columns of [VEC_GRID x ncols] partials into out, four columns' loads in flight a warp.
__device__ __forceinline__ void cta_col_sums(const double* part, int ncols, double* out) {
    constexpr int NP = (VEC_GRID + 31) / 32, NC = 4;
    const int lane = int(threadIdx.x & 31), w = int(threadIdx.x >> 5), nw = int(blockDim.x >> 5);
    for (int c0 = w; c0 < ncols; c0 += NC * nw) {
        double v[NC][NP];
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int i = 0; i < NP; i++) {
                const int col = c0 + c * nw, p = lane + 32 * i;
                v[c][i] = (col < ncols && p < VEC_GRID) ? __ldcg(part + size_t(p) * ncols + col) : 0.0;
            }
#pragma unroll
        for (int c = 0; c < NC; c++) {
            double acc = 0.0;
#pragma unroll
            for (int i = 0; i < NP; i++)
                if (lane + 32 * i < VEC_GRID) acc += v[c][i];
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
            if (lane == 0 && c0 + c * nw < ncols) out[c0 + c * nw] = acc;
        }
    }
}

// Per-CTA partials of a'b per column.
template <class T>
__device__ __forceinline__ void dot_partials(const T* __restrict__ a, const T* __restrict__ b, u32 m, int R,
                                             double* __restrict__ cta_part, double* red) {
    for (int j0 = 0; j0 < R; j0 += RC_MAX) {
        const ColMap cm = colmap(R, j0);
        double acc = 0.0;
        if (cm.on) {
#pragma unroll 4
            for (u32 i = blockIdx.x * u32(cm.nslot) + u32(cm.slot); i < m; i += gridDim.x * u32(cm.nslot)) {
                const size_t o = size_t(i) * R + j0 + cm.col;
                acc += double(a[o]) * double(b[o]);
            }
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        if (int(threadIdx.x) < cm.Rc) {
            double s = 0.0;
#pragma unroll 8
            for (int sl = 0; sl < cm.nslot; sl++) s += red[sl * cm.Rc + threadIdx.x];
            cta_part[size_t(blockIdx.x) * R + j0 + threadIdx.x] = s;
        }
        __syncthreads();
    }
}

// p'q, then gamma = rho / p'q on the active columns (a non-positive or non-finite p'q deactivates).
template <class T>
__global__ void __launch_bounds__(TB) k_pq_gamma(const T* __restrict__ p, const T* __restrict__ q, u32 m, int R,
                                                 double* __restrict__ cta_part, CgState st, CgLoop lp) {
    __shared__ double red[TB], fin[WIDE_R];
    if (__ldcg(lp.halt)) return;
    dot_partials(p, q, m, R, cta_part, red);
    const int j = int(threadIdx.x);
    double rho = 0.0, pfl = 0.0;
    int act = 0;
    if (j < R) {
        rho = st.rho[j];
        pfl = st.pfloor[j];
        act = st.active[j];
    }
    if (!last_of(lp.ticket, gridDim.x)) return;
    cta_col_sums(cta_part, R, fin);
    __syncthreads();
    if (j < R) {
        double g = 0.0;
        if (act == 1) {
            const double pq = fin[j];
            if (pq > 0.0 && isfinite(pq)) g = rho / pq;
            else st.active[j] = pfl > 0.0 ? 2 : 0;  // inner rounds: FP64 restart, not a stop
        }
        st.gamma[j] = g;
    }
}

// x += gamma p, r -= gamma q, and x'rhs, x'r, x0'r (x0 null: 0) into st.xb; with JACOBI also
// z = inv_diag r on the rows from ms on.
template <class T, bool JACOBI>
__global__ void __launch_bounds__(TB) k_update_xr(T* __restrict__ x, T* __restrict__ r, const T* __restrict__ p,
                                                  const T* __restrict__ q, const T* __restrict__ rhs,
                                                  const T* __restrict__ x0, u32 m, int R,
                                                  double* __restrict__ cta_part, CgState st, CgLoop lp,
                                                  T* __restrict__ z, const double* __restrict__ inv_diag, u32 ms) {
    __shared__ double red[3 * TB];
    if (__ldcg(lp.halt)) return;
    for (int j0 = 0; j0 < R; j0 += RC_MAX) {
        const ColMap cm = colmap(R, j0);
        double xb = 0.0, xr = 0.0, x0r = 0.0;
        if (cm.on) {
            const T g = T(st.gamma[j0 + cm.col]);
#pragma unroll 4
            for (u32 i = blockIdx.x * u32(cm.nslot) + u32(cm.slot); i < m; i += gridDim.x * u32(cm.nslot)) {
                const size_t o = size_t(i) * R + j0 + cm.col;
                const T xv = x[o] + g * p[o];
                const T rv = r[o] - g * q[o];
                x[o] = xv;
                r[o] = rv;
                xb += double(xv) * double(rhs[o]);
                xr += double(xv) * double(rv);
                if (x0) x0r += double(x0[o]) * double(rv);
                if (JACOBI && i >= ms) z[o] = T(__ldg(inv_diag + i)) * rv;
            }
        }
        red[threadIdx.x] = xb;
        red[TB + threadIdx.x] = xr;
        red[2 * TB + threadIdx.x] = x0r;
        __syncthreads();
        if (int(threadIdx.x) < 3 * cm.Rc) {  // thread (sum, column)
            const int v = int(threadIdx.x) / cm.Rc, c = int(threadIdx.x) % cm.Rc;
            double s = 0.0;
#pragma unroll 8
            for (int sl = 0; sl < cm.nslot; sl++) s += red[v * TB + sl * cm.Rc + c];
            cta_part[size_t(blockIdx.x) * 3 * R + v * R + j0 + c] = s;
        }
        __syncthreads();
    }
    if (!last_of(lp.ticket + 1, gridDim.x)) return;
    cta_col_sums(cta_part, 3 * R, st.xb);
}

// rho_new = r'z, then the stopping rule and beta. START: the rho of a (re)start instead
// (cg.rs:201-205): columns with rho <= 0 stop, the precision floor is drop rho, the active columns
// are counted.
template <class T, bool START>
__global__ void __launch_bounds__(TB) k_rz_stop(const T* __restrict__ r, const T* __restrict__ z, u32 m, int R,
                                                double* __restrict__ cta_part, CgState st, CgLoop lp, int probe_from,
                                                int probe_at, double drop) {
    __shared__ double red[TB], fin[WIDE_R];
    if (!START && __ldcg(lp.halt)) return;
    dot_partials(r, z, m, R, cta_part, red);
    const int j = int(threadIdx.x);
    ColState cs;
    double xsum = 0.0;
    if (!START && j < R) {
        cs.load(st, lp, j);
        xsum = cs.xconst + st.xb[j] + st.xb[R + j] + st.xb[2 * R + j];
    }
    if (!last_of(lp.ticket + 2, gridDim.x)) return;
    cta_col_sums(cta_part, R, fin);
    __syncthreads();
    bool live = false;
    if (j < R) {
        if (START) {
            st.rho[j] = fin[j];
            if (st.active[j] == 1 && !(fin[j] > 0.0)) st.active[j] = 0;
            st.pfloor[j] = drop * fin[j];
            live = st.active[j] == 1;
        } else {
            live = stop_column(st, lp, j, cs, fin[j], xsum, probe_from, probe_at);
        }
    }
    const int n = __syncthreads_count(live);
    if (threadIdx.x == 0) tile_done(st, lp, START ? 0 : cs.k, unsigned(n));
}

// The start of a batch of iterations (in a graph, a node before the WHILE node, whose first condition
// it sets): halt unless some column is active and the batch's cap allows an iteration.
__global__ void k_loop_first(cudaGraphConditionalHandle cond, int use_cond, const int* __restrict__ n_active, CgLoop lp) {
    if (threadIdx.x == 0) {
        const bool go = *n_active > 0 && lp.ctl[3] > 0;
        lp.ctl[4] = !go;
        if (use_cond) cudaGraphSetConditional(cond, go ? 1u : 0u);
    }
}

// p = z + beta p on the active columns, 0 on the others (START: p = z on the active ones); then the
// iteration's end: the launch's iteration count rises, the halt word is set where no further one may
// run, and the last iteration of a graph's body (use_cond) sets the WHILE condition.
template <class T, bool START>
__global__ void __launch_bounds__(TB) k_update_p(T* __restrict__ p, const T* __restrict__ z,
                                                 const double* __restrict__ beta, const int* __restrict__ active,
                                                 u32 m, int R, CgLoop lp, cudaGraphConditionalHandle cond,
                                                 int use_cond) {
    if (!START && __ldcg(lp.halt)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (lp.halt_next) *lp.halt_next = 1;
            if (use_cond) cudaGraphSetConditional(cond, 0u);
        }
        return;
    }
    const u32 Q = u32(R) / 4;
    const size_t total = size_t(m) * Q, step = size_t(gridDim.x) * TB;
    for (size_t i = size_t(blockIdx.x) * TB + threadIdx.x; i < total; i += step) {
        const u32 j = 4 * u32(i % Q);
        const V4<T> zv = ld4(z + 4 * i);
        V4<T> pv{T(0), T(0), T(0), T(0)};
        if (START) {
            if (active[j] == 1) pv.a = zv.a;
            if (active[j + 1] == 1) pv.b = zv.b;
            if (active[j + 2] == 1) pv.c = zv.c;
            if (active[j + 3] == 1) pv.d = zv.d;
        } else {
            const V4<T> o = ldv(p + 4 * i);
            if (active[j] == 1) pv.a = zv.a + T(beta[j]) * o.a;
            if (active[j + 1] == 1) pv.b = zv.b + T(beta[j + 1]) * o.b;
            if (active[j + 2] == 1) pv.c = zv.c + T(beta[j + 2]) * o.c;
            if (active[j + 3] == 1) pv.d = zv.d + T(beta[j + 3]) * o.d;
        }
        st4(p + 4 * i, pv);
    }
    if (!START && blockIdx.x == 0 && threadIdx.x == 0) {
        const int kl = ++lp.ctl[2];
        const bool go = lp.ctl[0] > 0 && kl < lp.ctl[3];
        if (lp.halt_next) *lp.halt_next = !go;  // another word than the one the other CTAs still read
        if (use_cond) cudaGraphSetConditional(cond, go ? 1u : 0u);
    }
}

}  // namespace fereg
