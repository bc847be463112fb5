// dpf_gpersist.cuh -- a whole CG + AMG solve on a face list (CSR) as one cooperative launch, the
// counterpart of dpf_persist.cuh: one block per SM, grid barriers between the steps, every block forming
// the CG scalars for itself, convergence decided on the device. The host-driven loop took about 50
// launches per iteration and a synchronisation for each convergence read: 386 us per iteration for a
// fracture network of 815k cells in mixed precision, 335 us for 200k cells in FP64; now 205 us and 140 us
// (a forward and adjoint of the network 72 -> 43 ms, Richards' Picard and adjoint solves 63 -> 32 ms).
// The finest level's steps are near the memory's rate (9..17 us each: gathers through the column indices);
// a step on a small level takes 3..4 us, of which a barrier is 1.3. Those steps are bound by trips to L2:
// a block keeps its rows of the small levels in shared memory, 2 to 8 lanes (FP64: 4) share a row, and the ranges of
// a block's rows are worked out once (they cost two integer divisions per step). Together 51.3 -> 44.3 ms
// and 34.3 -> 31.3 ms.
//
// Per level the rows are cut into equal contiguous shares of whole groups of 32, one per block; the levels
// of a few hundred cells run in one block. The first smoothing pass reads u = b D^-1, stored by the pass
// that makes b, instead of two gathers per coupling; FP64 levels form b - A x as b - a_ii x_i + sum c x_j
// (one FP64 instruction per coupling, CG's own products keep the flux form) and keep the Chebyshev direction
// as e = D d.
#pragma once
#include "dpf_grid.cuh"

namespace dpf {

constexpr int kGpThreads = 1024;
constexpr int kGpLevels = 24;
constexpr int kGpTail = 512;   // cells of the one-block tail's first level (256: 3 % slower, 1024: the same)
constexpr int kGpRowBytes = 64 * 1024;  // shared memory for the rows' copies (144 KB: 0.9 % slower, L1 is smaller)

template <typename T>
struct GpLevel {
    int n;
    const int *rp, *ci, *agg, *mrp, *mci;
    const T *v, *leak, *idg, *dg;  // dg: FP64 only
    T *xa, *xb, *b, *d, *u;
    const uint8_t *dir;
};

template <typename T>
struct GpParams {
    GpLevel<T> lv[kGpLevels];
    int nl, tail, deg, dense;      // tail: first level of the one-block tail (nl: none)
    T c1[8], c2[8], e1[8], e2[8], invtheta, scale;  // e1, e2: the degree-8 sweep of a coarsest level that is not dense
    const double *Inv;
    CgState *st;
    unsigned *bar;
    int *expired;
    double2 *partials;             // two halves of one slot per block
    double tol2;
    int maxiter, max_rounds, row_bytes;
    const uint8_t *dir;
    const double *b64;
    double *x64;
    T *r, *z;
    double *p, *q;                 // FP64 CG
    double *r64;                   // mixed
    float2 *rd, *pd, *qd;
    const float2 *vdf, *leakdf;
    const double *v64, *leak64;    // finest couplings in FP64
};

// (A x)_i in flux form with the FP64 couplings of the finest level; the diagonal beside it
__device__ __forceinline__ double gp_flux(int n, const int *rp, const int *ci, const double *v, const double *leak, int i,
                                          double xi, const double *x, double &diag) {
    const double lk = leak[i];
    double a = lk * xi, d = lk;
    const int e1 = rp[i + 1];
    for (int e = rp[i]; e < e1; e++) {
        const double w = v[e];
        if (!DPF_INSIDE(CK_ONE_COL, ci[e], 0, n)) continue;
        a += w * (xi - x[ci[e]]);
        d += w;
    }
    diag = d;
    return a;
}

// The rows that this block works on, indexed as the whole arrays are: its shared-memory copies where they
// fit, the arrays themselves where they do not.
template <typename T>
struct GpRows {
    const int *rp, *ci;
    const T *v;
    const int *mrp, *mci;  // members of the rows' aggregates (rows of the level below the first)
    const int *aci;        // the aggregates of the columns (null: not copied)
    T *xa, *xb, *b, *d, *u;  // the level's vectors: the whole arrays, or the tail's block's own copies
    int i0, i1, lg;        // this block's rows, and 1 << lg lanes to a row where the level is small
    bool small;
};
// 1 << lg lanes of a warp share a row; q is this thread's place among them
struct GpLane {
    int lg, q;
    template <typename A>
    __device__ __forceinline__ A sum(A a) const {
        for (int o = (1 << lg) >> 1; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        return a;
    }
};

// b_i - (A x)_i of a V-cycle level, in every lane of the row; FP32: also the diagonal, for the smoother's
// division. kSmall: a row of R shared by the lanes of ln; otherwise a row of the level's arrays, by one thread.
// x(e, j): the value at entry e's column j.
template <bool kSmall, typename T, typename X>
__device__ __forceinline__ T gp_resid(const GpLevel<T> &V, const GpRows<T> &R, GpLane ln, int i, T bi, T xi, X x,
                                      T &diag) {
    const int *rp = kSmall ? R.rp : V.rp, *ci = kSmall ? R.ci : V.ci;
    const T *v = kSmall ? R.v : V.v;
    const int e1 = rp[i + 1], by = kSmall ? 1 << ln.lg : 1;
    if constexpr (sizeof(T) == 8) {
        T r = kSmall ? T(0) : fma(-V.dg[i], xi, bi);
        diag = T(0);
        for (int e = rp[i] + (kSmall ? ln.q : 0); e < e1; e += by)
            if (DPF_INSIDE(CK_ONE_COL, ci[e], 0, V.n)) r = fma(v[e], x(e, ci[e]), r);
        return kSmall ? fma(-V.dg[i], xi, bi) + ln.sum(r) : r;
    } else {
        const T lk = V.leak[i];
        T a = kSmall ? T(0) : lk * xi, d = kSmall ? T(0) : lk;
        for (int e = rp[i] + (kSmall ? ln.q : 0); e < e1; e += by) {
            const T w = v[e];
            if (!DPF_INSIDE(CK_ONE_COL, ci[e], 0, V.n)) continue;
            a += w * (xi - x(e, ci[e]));
            d += w;
        }
        diag = kSmall ? lk + ln.sum(d) : d;
        return bi - (kSmall ? fma(lk, xi, ln.sum(a)) : a);
    }
}

template <typename T>
struct GpSolve {
    // Small levels, FP32: the prolongation is part of the first smoothing step after it (not of one that ends
    // the cycle). One step less per level (a network of 815k cells 45.6 -> 44.4 ms); in FP64 the products it
    // adds to every coupling cost as much as the step.
    static constexpr bool kFuse = sizeof(T) == 4;
    const GpParams<T> &P;
    GridBar bar;
    CgState &s;        // shared memory, the same in every block
    GpRows<T> *rw;     // shared memory: this block's rows of every level
    int half;

    __device__ __forceinline__ double2 *slots() const { return P.partials + (half ? gridDim.x : 0); }
    // this block's rows of a level of n, or all of them (one: the tail's block)
    __device__ __forceinline__ static void rows(int n, bool one, int &i0, int &i1) {
        i0 = 0;
        i1 = n;
        if (one) return;
        const int units = (n + 31) >> 5, k = gridDim.x, base = units / k, more = units - base * k, q = blockIdx.x;
        i0 = min(n, 32 * (q * base + min(q, more)));
        i1 = min(n, 32 * ((q + 1) * base + min(q + 1, more)));
    }
    // this block's rows of the finest level
    template <typename F>
    __device__ __forceinline__ void each(F f) const {
        const int i1 = rw[0].i1;
#pragma unroll 1
        for (int i = rw[0].i0 + (int)threadIdx.x; i < i1; i += kGpThreads) f(i);
    }
    // Does a block have so few rows of a level of n that several lanes share one?
    __device__ __forceinline__ static bool small(int n, bool one) {
        return one || 64 * (((n + 31) / 32 + (int)gridDim.x - 1) / (int)gridDim.x) <= kGpThreads;
    }
    // log2 of the lanes to a row where a block has m: at most 8, in FP64 at most 4 (the sums between the lanes are
    // FP64 instructions too: 200k cells of Richards' equation 28.9 ms with 8, 28.1 with 4, 29.7 with 2, 35.4 with 1;
    // a network of 815k mixed cells 45.1 ms with 4, 44.5 with 8, 44.4 with 16)
    __device__ __forceinline__ static int lanes(int m) {
        int lg = 0;
        while (lg < (sizeof(T) == 8 ? 2 : 3) && (m << (lg + 1)) <= kGpThreads) lg++;
        return lg;
    }
    // Rows i0 .. i1 - 1. kSmall: 2 to 8 lanes to a row, f(row, lane, whether this thread stores the row's
    // results) with all lanes of a warp: a thread gathers a row's entries four at a time, each time a trip
    // to L2.
    template <bool kSmall, typename F>
    __device__ __forceinline__ static void each_row(int i0, int i1, int lg, F f) {
        if constexpr (!kSmall) {
#pragma unroll 1
            for (int i = i0 + (int)threadIdx.x; i < i1; i += kGpThreads) f(i, GpLane{0, 0}, true);
        } else {
            const GpLane ln{lg, (int)threadIdx.x & ((1 << lg) - 1)};
#pragma unroll 1
            for (int b = i0; b + ((int)(threadIdx.x & ~31u) >> lg) < i1; b += kGpThreads >> lg) {
                const int i = b + ((int)threadIdx.x >> lg);
                f(min(i, i1 - 1), ln, i < i1 && ln.q == 0);
            }
        }
    }
    // Shared-memory copies of this block's rows of the small levels, coarsest first, while they fit: a step
    // then waits for one trip to L2, its gathers, instead of three (row pointers, columns, gathers). In the
    // tail's block also the tail's vectors, except those of its first level that other blocks write or read.
    __device__ __forceinline__ void stage_rows(unsigned char *mem, int bytes) {
        int used = 0;
#pragma unroll 1
        for (int l = P.nl - 1; l >= 0; l--) {
            const GpLevel<T> &V = P.lv[l];
            const bool one = l >= P.tail, mem_rows = l > P.tail || (l > 0 && !one);  // with their members
            int i0 = 0, i1 = 0;
            if (!one || blockIdx.x == 0) rows(V.n, one, i0, i1);
            const int m = i1 - i0;
            GpRows<T> r{V.rp, V.ci, V.v, l ? P.lv[l - 1].mrp : nullptr, l ? P.lv[l - 1].mci : nullptr, nullptr,
                        V.xa, V.xb, V.b, V.d, V.u, i0, i1, lanes(m), small(V.n, one)};
            if (m > 0 && r.small) {
                const int e0 = V.rp[i0], ne = V.rp[i1] - e0;
                const int a0 = mem_rows ? r.mrp[i0] : 0, na = mem_rows ? r.mrp[i1] - a0 : 0;
                const int nv = !one ? 0 : l == P.tail ? 2 : 5;
                const int nag = kFuse && l + 1 < P.nl ? ne : 0;
                const int need = ((ne + nv * m) * (int)sizeof(T) + 4 * (ne + nag + (mem_rows ? 2 : 1) * (m + 1) + na) + 15) & ~15;
                if (used + need <= bytes) {
                    T *v = (T *)(mem + used), *vec = v + ne;
                    int *ci = (int *)(vec + nv * m), *aci = ci + ne, *rp = aci + nag, *mrp = rp + m + 1, *mci = mrp + m + 1;
                    for (int k = threadIdx.x; k < ne; k += kGpThreads) {
                        v[k] = V.v[e0 + k];
                        const int j = V.ci[e0 + k];
                        ci[k] = j;
                        if (nag) aci[k] = DPF_INSIDE(CK_ONE_COL, j, 0, V.n) ? V.agg[j] : -1;
                    }
                    for (int k = threadIdx.x; k <= m; k += kGpThreads) {
                        rp[k] = V.rp[i0 + k];
                        if (mem_rows) mrp[k] = r.mrp[i0 + k];
                    }
                    for (int k = threadIdx.x; k < na; k += kGpThreads) mci[k] = r.mci[a0 + k];
                    r.rp = rp - i0;
                    r.ci = ci - e0;
                    r.v = v - e0;
                    if (nag) r.aci = aci - e0;
                    if (mem_rows) {
                        r.mrp = mrp - i0;
                        r.mci = mci - a0;
                    }
                    if (one) {
                        r.xa = vec;
                        r.d = vec + m;
                        if (l > P.tail) {
                            r.xb = vec + 2 * m;
                            r.b = vec + 3 * m;
                            r.u = vec + 4 * m;
                        }
                    }
                    used += need;
                }
            }
            if (threadIdx.x == 0) rw[l] = r;
        }
        __syncthreads();
    }
    // the step's barrier: the grid's, or the block's in the tail
    __device__ __forceinline__ bool step(bool one) {
        if (!one) return bar.sync();
        __syncthreads();
        return true;
    }
    // sums of a and b over all blocks, then f(total) in one thread of every block
    template <typename A, int NV, typename F>
    __device__ __forceinline__ bool reduce(Acc<A> a, Acc<A> b, F f) {
        const double2 t = block_sum<A, NV>(a, b);
        if (threadIdx.x == 0) slots()[blockIdx.x] = t;
        if (!bar.sync()) return false;
        if (threadIdx.x < 32) {
            double2 t = make_double2(0.0, 0.0);
#pragma unroll 1
            for (int k = threadIdx.x; k < (int)gridDim.x; k += 32) {
                const double2 v = __ldcg(slots() + k);
                t.x += v.x;
                if (NV == 2) t.y += v.y;
            }
            t.x = warp_sum(t.x);
            if (NV == 2) t.y = warp_sum(t.y);
            if (threadIdx.x == 0) f(t);
        }
        half ^= 1;  // a slower block may still be reading this half
        __syncthreads();
        return true;
    }
    __device__ __forceinline__ void set_beta(double rz) {
        s.rz_old = s.rz;
        s.rz = rz;
        s.beta = (s.iters == 0 || s.rz_old == 0.0) ? 0.0 : s.rz / s.rz_old;
    }
    __device__ __forceinline__ void put_r(int i, T r) const {
        P.r[i] = r;
        P.lv[0].u[i] = r * P.lv[0].idg[i];
    }

    // Chebyshev step k of a sweep with coefficients (k1, k2) from cur to o; FIRST: no direction before it
    template <bool kSmall, bool FIRST, bool DOT>
    __device__ __forceinline__ Acc<T> cheb(int l, const T *b, const T *cur, T *o, T k1, T k2) {
        const GpLevel<T> &V = P.lv[l];
        const GpRows<T> R = rw[l];
        T *const d = kSmall ? R.d : V.d;
        Acc<T> a;
        each_row<kSmall>(R.i0, R.i1, R.lg, [&](int i, GpLane ln, bool store) {
            T xi = cur[i], dg;
            const T bi = b[i];
            T r;
            if constexpr (kSmall && FIRST && kFuse) {
                const T *e = rw[l + 1].xb;
                auto corr = [&](int a) {
                    return a >= 0 && DPF_INSIDE(CK_ONE_AGG, a, 0, P.lv[l + 1].n) ? P.scale * e[a] : T(0);
                };
                if (!V.dir[i]) xi += corr(V.agg[i]);
                // coupled cells are free cells
                r = gp_resid<true>(V, R, ln, i, bi, xi,
                                   [&](int k, int j) { return cur[j] + corr(R.aci ? R.aci[k] : V.agg[j]); }, dg);
            } else {
                r = gp_resid<kSmall>(V, R, ln, i, bi, xi, [&](int, int j) { return cur[j]; }, dg);
            }
            T dn, xo;
            if constexpr (sizeof(T) == 8) {
                dn = FIRST ? k2 * r : fma(k2, r, k1 * d[i]);
                xo = fma(V.idg[i], dn, xi);
            } else {
                const T rd = __fdividef(r, dg);
                dn = FIRST ? k2 * rd : k1 * d[i] + k2 * rd;
                xo = xi + dn;
            }
            if (!store) return;
            d[i] = dn;
            o[i] = xo;
            if (DOT) a = a + Acc<T>::prod(bi, xo);
        });
        return a;
    }
    // the first step from a zero guess (into xa), or the first two (into xb)
    template <bool kSmall>
    __device__ __forceinline__ void first(int l, const T *b, bool two, T k1, T k2) {
        const GpLevel<T> &V = P.lv[l];
        const GpRows<T> R = rw[l];
        T *const d = kSmall ? R.d : V.d, *const xa = kSmall ? R.xa : V.xa, *const xb = kSmall ? R.xb : V.xb;
        const T *u = kSmall ? R.u : V.u;
        if (!two) {
            each_row<false>(R.i0, R.i1, 0, [&](int i, GpLane, bool) {
                const T x1 = P.invtheta * u[i];
                d[i] = sizeof(T) == 8 ? P.invtheta * b[i] : x1;
                xa[i] = x1;
            });
            return;
        }
        each_row<kSmall>(R.i0, R.i1, R.lg, [&](int i, GpLane ln, bool store) {
            const T ui = u[i], x1 = P.invtheta * ui;
            T dg;
            const T t = gp_resid<kSmall>(V, R, ln, i, T(0), ui, [&](int, int j) { return u[j]; }, dg);  // -(A u)_i
            const T bi = b[i], r = fma(P.invtheta, t, bi);
            if (!store) return;
            if constexpr (sizeof(T) == 8) {
                const T e = fma(k2, r, k1 * P.invtheta * bi);
                d[i] = e;
                xb[i] = fma(V.idg[i], e, x1);
            } else {
                const T dn = k1 * x1 + k2 * r * V.idg[i];
                d[i] = dn;
                xb[i] = x1 + dn;
            }
        });
    }
    template <bool kSmall>
    __device__ __forceinline__ void residual(int l, const T *b, const T *cur) {
        const GpLevel<T> &V = P.lv[l];
        const GpRows<T> R = rw[l];
        T *const d = kSmall ? R.d : V.d;
        each_row<kSmall>(R.i0, R.i1, R.lg, [&](int i, GpLane ln, bool store) {
            T dg;
            const T r = gp_resid<kSmall>(V, R, ln, i, b[i], cur[i], [&](int, int j) { return cur[j]; }, dg);
            if (store) d[i] = r;
        });
    }
    // the members' sums of every aggregate of level l (in member order, or lane by lane) to level l + 1
    template <bool kSmall>
    __device__ __forceinline__ void restrict_to(int l, bool one) {
        const GpLevel<T> &V = P.lv[l], &W = P.lv[l + 1];
        const GpRows<T> R = rw[l + 1];
        const bool in_rows = kSmall && (one || l + 1 < P.tail);
        const int *mrp = in_rows ? R.mrp : V.mrp, *mci = in_rows ? R.mci : V.mci;
        const T *d = rw[l].d;
        int i0 = R.i0, i1 = R.i1, lg = R.lg;
        if (kSmall && !in_rows) {  // the tail's first level, by all blocks
            rows(W.n, false, i0, i1);
            lg = lanes(i1 - i0);
        }
        each_row<kSmall>(i0, i1, lg, [&](int I, GpLane ln, bool store) {
            T a = 0;
            const int k1 = mrp[I + 1];
            for (int k = mrp[I] + ln.q; k < k1; k += 1 << ln.lg)
                if (DPF_INSIDE(CK_ONE_AGG, mci[k], 0, V.n)) a += d[mci[k]];
            if (kSmall) a = ln.sum(a);
            if (!store) return;
            R.b[I] = a;
            R.u[I] = a * W.idg[I];
        });
    }
    // a smoothing step of any level
    template <bool FIRST>
    __device__ __forceinline__ void smooth(int l, const T *b, const T *cur, T *o, T k1, T k2, bool sm) {
        if (sm) cheb<true, FIRST, false>(l, b, cur, o, k1, k2);
        else cheb<false, FIRST, false>(l, b, cur, o, k1, k2);
    }

    // z = M r; ends with r . z and beta
    __device__ __forceinline__ bool vcycle() {
        const int deg = P.deg;
        bool mine = true;  // does this block work on the levels at hand?
#pragma unroll 1
        for (int l = 0; l < P.nl; l++) {
            const GpLevel<T> &V = P.lv[l];
            const bool one = l >= P.tail, sm = rw[l].small;
            if (one && blockIdx.x != 0) {
                mine = false;
                break;
            }
            T *const xa = rw[l].xa, *const xb = rw[l].xb;
            const T *b = l == 0 ? P.r : rw[l].b;
            if (l == P.nl - 1) {
                T *out = l == 0 ? P.z : xb;
                if (P.dense) {
                    // eight lanes per row of the stored inverse; by one block
                    if (blockIdx.x == 0 && threadIdx.x < 8 * kMaxCoarse) {
                        const int i = threadIdx.x >> 3, q = threadIdx.x & 7;
                        double x = 0.0;
                        if (i < V.n)
                            for (int j = q; j < V.n; j += 8) x = fma(P.Inv[j * kMaxCoarse + i], (double)b[j], x);
#pragma unroll
                        for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                        if (i < V.n && q == 0) out[i] = (T)x;
                    }
                } else {
                    // no useful coarsening left: a degree-8 sweep stands in for the solve
                    if (sm) first<true>(l, b, false, T(0), T(0));
                    else first<false>(l, b, false, T(0), T(0));
                    if (!step(one)) return false;
                    T *cur = xa;
#pragma unroll 1
                    for (int k = 1; k < 8; k++) {
                        T *o = k == 7 ? out : (cur == xa ? xb : xa);
                        if (o == cur) o = cur == xa ? xb : xa;
                        smooth<false>(l, b, cur, o, P.e1[k], P.e2[k], sm);
                        if (!step(one)) return false;
                        cur = o;
                    }
                }
                if (!step(one)) return false;
                break;
            }
            T *cur = deg >= 2 ? xb : xa;
            const T f1 = deg >= 2 ? P.c1[1] : T(0), f2 = deg >= 2 ? P.c2[1] : T(0);
            if (sm) first<true>(l, b, deg >= 2, f1, f2);
            else first<false>(l, b, deg >= 2, f1, f2);
            if (!step(one)) return false;
#pragma unroll 1
            for (int k = 2; k < deg; k++) {
                T *o = cur == xa ? xb : xa;
                smooth<false>(l, b, cur, o, P.c1[k], P.c2[k], sm);
                if (!step(one)) return false;
                cur = o;
            }
            if (sm) residual<true>(l, b, cur);
            else residual<false>(l, b, cur);
            if (!step(one)) return false;
            if (rw[l + 1].small) restrict_to<true>(l, one);
            else restrict_to<false>(l, one);
            // the tail's block reads what the others wrote, and they wait for its last barrier
            if (!(one ? step(true) : bar.sync())) return false;
        }
#pragma unroll 1
        for (int l = P.nl - 2; l >= 0; l--) {
            const GpLevel<T> &V = P.lv[l];
            const bool one = l >= P.tail, sm = rw[l].small;
            if (one && !mine) continue;
            if (!one && l + 1 >= P.tail && !bar.sync()) return false;  // the tail is done
            T *const xa = rw[l].xa, *const xb = rw[l].xb;
            const T *b = l == 0 ? P.r : rw[l].b, *e = rw[l + 1].xb;
            // where pre-smoothing left its iterate
            T *cur = (deg % 2 == 0) ? xb : xa;
            if (!kFuse || !sm || (l == 0 && deg == 1)) {
                each_row<false>(rw[l].i0, rw[l].i1, 0, [&](int i, GpLane, bool) {
                    const int a = V.agg[i];
                    if (a >= 0 && !V.dir[i] && DPF_INSIDE(CK_ONE_AGG, a, 0, P.lv[l + 1].n)) cur[i] += P.scale * e[a];
                });
                if (!step(one)) return false;
            }
#pragma unroll 1
            for (int k = 0; k < deg; k++) {
                const bool rz = k == deg - 1 && l == 0;
                T *o = rz ? P.z : (cur == xa ? xb : xa);
                if (rz) {
                    const Acc<T> a = k == 0 ? cheb<false, true, true>(l, b, cur, o, T(0), P.invtheta)
                                            : cheb<false, false, true>(l, b, cur, o, P.c1[k], P.c2[k]);
                    if (!reduce<T, 1>(a, Acc<T>(), [&](double2 t) { set_beta(t.x); })) return false;
                } else {
                    if (k == 0) smooth<true>(l, b, cur, o, T(0), P.invtheta, sm);
                    else smooth<false>(l, b, cur, o, P.c1[k], P.c2[k], sm);
                    if (!step(one)) return false;
                }
                cur = o;
            }
        }
        if (P.nl == 1) {  // no smoothing pass: the coarsest solve's r . z
            Acc<double> a;
            each([&](int i) { a.v += (double)P.r[i] * (double)P.z[i]; });
            if (!reduce<double, 1>(a, Acc<double>(), [&](double2 t) { set_beta(t.x); })) return false;
        }
        return true;
    }
    __device__ __forceinline__ void end_iteration(double rr, bool met, int iters) {
        s.rr = rr;
        s.iters++;
        s.total_iters++;
        if (!isfinite(rr)) s.status = DPF_NAN;
        else if (met) {}
        else if (iters + 1 >= P.maxiter) s.status = DPF_NOT_CONVERGED;
        else return;
        s.active = 0;
    }
    __device__ __forceinline__ void set_alpha(double pq) {
        s.pq = pq;
        s.alpha = 0.0;
        if (!isfinite(pq)) s.status = DPF_NAN;
        else if (pq > 0.0) {
            s.alpha = s.rz / pq;
            return;
        }
        s.active = 0;  // p = 0: exact solution
    }
    __device__ __forceinline__ void start(double rr, double bb, bool go) {
        s.tol2 = P.tol2;
        s.status = DPF_OK;
        if (!isfinite(rr)) {
            s.status = DPF_NAN;
            go = false;
        }
        s.active = go ? 1 : 0;
    }

    __device__ __forceinline__ void run(unsigned char *mem) {
        const int *rp = P.lv[0].rp, *ci = P.lv[0].ci;
        if constexpr (sizeof(T) == 8) {
            const double *v = P.v64;
            Acc<double> rr, bb;
            each([&](int i) {
                double dg;
                const double bi = P.b64[i];
                const double ri = bi - gp_flux(P.lv[0].n, rp, ci, v, P.leak64, i, P.x64[i], P.x64, dg);
                put_r(i, ri);
                rr.v += ri * ri;
                if (!P.dir[i]) bb.v += bi * bi;
            });
            if (!reduce<double, 2>(rr, bb, [&](double2 t) {
                    s.rr = t.x;
                    s.bb = t.y;
                    start(t.x, t.y, t.y > 0.0 && t.x > P.tol2 * t.y);
                }))
                return;
            if (!s.active) return;
            stage_rows(mem, P.row_bytes);
            for (int it = 0;; it++) {
                if (!vcycle()) return;
                const double beta = s.beta;
                each([&](int i) { P.p[i] = beta == 0.0 ? P.z[i] : P.z[i] + beta * P.p[i]; });
                if (!bar.sync() || it > P.maxiter) return;
                Acc<double> a;
                each([&](int i) {
                    double dg;
                    const double pi = P.p[i], qi = gp_flux(P.lv[0].n, rp, ci, v, P.leak64, i, pi, P.p, dg);
                    P.q[i] = qi;
                    a.v += pi * qi;
                });
                if (!reduce<double, 1>(a, Acc<double>(), [&](double2 t) { set_alpha(t.x); })) return;
                if (!s.active) return;
                const double al = s.alpha;
                Acc<double> c;
                each([&](int i) {
                    P.x64[i] += al * P.p[i];
                    const double ri = P.r[i] - al * P.q[i];
                    put_r(i, ri);
                    c.v += ri * ri;
                });
                if (!reduce<double, 1>(c, Acc<double>(), [&](double2 t) {
                        end_iteration(t.x, t.x <= s.tol2 * s.bb, s.iters);
                    }))
                    return;
                if (!s.active) return;
            }
        } else {
            for (int round = -1; round < P.max_rounds; round++) {
                const bool fst = round < 0;
                Acc<double> rr, bb;  // first: |r|^2, |b|^2; later: |r|^2 and the rounding floor
                each([&](int i) {
                    double dg;
                    const double xi = P.x64[i], bi = P.b64[i];
                    const double ri = bi - gp_flux(P.lv[0].n, rp, ci, P.v64, P.leak64, i, xi, P.x64, dg);
                    P.r64[i] = ri;
                    rr.v += ri * ri;
                    if (P.dir[i]) return;  // identity row: in neither
                    if (fst) {
                        bb.v += bi * bi;
                    } else {
                        const double f = 0x1p-48 * fma(2.0 * dg, fabs(xi), fabs(bi));
                        bb.v += f * f;
                    }
                });
                if (!reduce<double, 2>(rr, bb, [&](double2 t) {
                        s.orr = t.x;
                        if (fst) {
                            s.obb = t.y;
                            start(t.x, t.y, t.y > 0.0 && t.x > P.tol2 * t.y);
                        } else {
                            s.outer++;
                            s.floor2 = t.y;
                            // at the FP64 rounding floor of b - A x: accepted (no further accuracy exists)
                            const bool floor = s.orr <= s.floor2 || s.orr > 0.25 * s.orr_prev;
                            s.active = 1;
                            if (!isfinite(s.orr)) { s.status = DPF_NAN; s.active = 0; }
                            else if (s.orr <= P.tol2 * s.obb || floor) s.active = 0;
                            else if (s.total_iters >= P.maxiter || s.outer >= P.max_rounds) {
                                s.status = DPF_NOT_CONVERGED;
                                s.active = 0;
                            }
                        }
                        s.orr_prev = s.orr;
                        s.iters = 0;
                        s.rz = s.rz_old = s.beta = 0.0;
                        if (s.active) s.scale = sqrt(s.orr);
                    }))
                    return;
                if (!s.active || round + 1 >= P.max_rounds) return;
                if (fst) stage_rows(mem, P.row_bytes);
                const double inv = 1.0 / s.scale, scale = s.scale;
                each([&](int i) {
                    const float2 v = df_from_double(P.r64[i] * inv);
                    P.rd[i] = v;
                    put_r(i, v.x);
                });
                if (!bar.sync()) return;
                for (int it = 0;; it++) {
                    if (!vcycle()) return;
                    const double beta = s.beta;
                    const float2 bd = df_from_double(beta);
                    each([&](int i) {
                        const float2 zi = make_float2(P.z[i], 0.0f);
                        P.pd[i] = beta == 0.0 ? zi : df_add(zi, df_mul(bd, P.pd[i]));
                    });
                    if (!bar.sync()) return;
                    if (it > P.maxiter) break;
                    Acc<float> a;
                    each([&](int i) {
                        const float2 pi = P.pd[i];
                        float2 v = df_mul(P.leakdf[i], pi);
                        const int e1 = rp[i + 1];
                        for (int e = rp[i]; e < e1; e++)
                            if (DPF_INSIDE(CK_ONE_COL, ci[e], 0, P.lv[0].n))
                                v = df_add(v, df_mul(P.vdf[e], df_sub(pi, P.pd[ci[e]])));
                        P.qd[i] = v;
                        a = a + Acc<float>::prod(pi.x, v.x);
                    });
                    if (!reduce<float, 1>(a, Acc<float>(), [&](double2 t) { set_alpha(t.x); })) return;
                    if (!s.active) break;
                    const float2 al = df_from_double(s.alpha);
                    const double as = s.alpha * scale;
                    Acc<float> c;
                    each([&](int i) {
                        const float2 pi = P.pd[i];
                        P.x64[i] = fma(as, (double)pi.x + (double)pi.y, P.x64[i]);
                        const float2 ri = df_sub(P.rd[i], df_mul(al, P.qd[i]));
                        P.rd[i] = ri;
                        put_r(i, ri.x);
                        c = c + Acc<float>::prod(ri.x, ri.x);
                    });
                    if (!reduce<float, 1>(c, Acc<float>(), [&](double2 t) {
                            end_iteration(t.x, t.x * s.scale * s.scale <= s.tol2 * s.obb || t.x <= kRoundDrop2,
                                          s.total_iters);
                        }))
                        return;
                    if (!s.active) break;
                }
                // a NaN or the iteration cap inside the round: the check keeps its status unless it passes
            }
        }
    }
};

template <typename T>
__global__ void __launch_bounds__(kGpThreads, 1) kg_solve_persistent(const __grid_constant__ GpParams<T> P) {
    __shared__ CgState st;
    __shared__ GpRows<T> rw[kGpLevels];
    extern __shared__ __align__(16) unsigned char gp_mem[];
    if (threadIdx.x == 0) {
        memset(&st, 0, sizeof(st));
        st.cont = 1.0;
        // what the first residual needs; the rest, and the copies, once there is something to iterate (a warm-started step
        // that is solved already: 54 -> 46 us, with separate launches 52)
        GpSolve<T>::rows(P.lv[0].n, false, rw[0].i0, rw[0].i1);
    }
    __syncthreads();
    GpSolve<T> S{P, GridBar{P.bar, P.expired}, st, rw, 0};
    S.run(gp_mem);
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) P.st[0] = st;
}

}  // namespace dpf
