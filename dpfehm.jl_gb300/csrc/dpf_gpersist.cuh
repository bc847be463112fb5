// dpf_gpersist.cuh -- a whole CG + AMG solve on a face list (CSR) as one cooperative launch, the
// counterpart of dpf_persist.cuh: one block per SM, grid barriers between the steps, every block forming
// the CG scalars for itself, convergence decided on the device. The host-driven loop took about 50
// launches per iteration and a synchronisation for each convergence read: 386 us per iteration for a
// fracture network of 815k cells in mixed precision, 335 us for 200k cells in FP64; now 239 us and 156 us
// (a forward and adjoint of the network 72.5 -> 48.9 ms, Richards' Picard and adjoint solves 62.9 -> 38.9 ms).
// Of the 239 us the finest level's steps take 9..17 us each (gathers through the column indices), the
// small levels ~4 us a step (a barrier is 1.5 us of it) and the one-block tail 25 us.
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
constexpr int kGpTail = 512;   // cells of the one-block tail's first level

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
    int maxiter, max_rounds;
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
__device__ __forceinline__ double gp_flux(const int *rp, const int *ci, const double *v, const double *leak, int i,
                                          double xi, const double *x, double &diag) {
    const double lk = leak[i];
    double a = lk * xi, d = lk;
    const int e1 = rp[i + 1];
    for (int e = rp[i]; e < e1; e++) {
        const double w = v[e];
        a += w * (xi - x[ci[e]]);
        d += w;
    }
    diag = d;
    return a;
}

// b_i - (A x)_i of a V-cycle level; FP32: also the diagonal, for the smoother's division
template <typename T>
__device__ __forceinline__ T gp_resid(const GpLevel<T> &V, int i, T bi, T xi, const T *x, T &diag) {
    const int e1 = V.rp[i + 1];
    if constexpr (sizeof(T) == 8) {
        T r = fma(-V.dg[i], xi, bi);
        diag = T(0);
        for (int e = V.rp[i]; e < e1; e++) r = fma(V.v[e], x[V.ci[e]], r);
        return r;
    } else {
        const T lk = V.leak[i];
        T a = lk * xi, d = lk;
        for (int e = V.rp[i]; e < e1; e++) {
            const T w = V.v[e];
            a += w * (xi - x[V.ci[e]]);
            d += w;
        }
        diag = d;
        return bi - a;
    }
}

template <typename T>
struct GpSolve {
    const GpParams<T> &P;
    GridBar bar;
    CgState &s;        // shared memory, the same in every block
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
    template <typename F>
    __device__ __forceinline__ static void each(int n, bool one, F f) {
        int i0, i1;
        rows(n, one, i0, i1);
#pragma unroll 1
        for (int i = i0 + (int)threadIdx.x; i < i1; i += kGpThreads) f(i);
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
    template <bool FIRST, bool DOT>
    __device__ __forceinline__ Acc<T> cheb(const GpLevel<T> &V, const T *b, const T *cur, T *o, T k1, T k2, bool one) {
        Acc<T> a;
        each(V.n, one, [&](int i) {
            const T xi = cur[i], bi = b[i];
            T dg;
            const T r = gp_resid(V, i, bi, xi, cur, dg);
            T dn, xo;
            if constexpr (sizeof(T) == 8) {
                dn = FIRST ? k2 * r : fma(k2, r, k1 * V.d[i]);
                xo = fma(V.idg[i], dn, xi);
            } else {
                const T rd = __fdividef(r, dg);
                dn = FIRST ? k2 * rd : k1 * V.d[i] + k2 * rd;
                xo = xi + dn;
            }
            V.d[i] = dn;
            o[i] = xo;
            if (DOT) a = a + Acc<T>::prod(bi, xo);
        });
        return a;
    }
    // the first step from a zero guess (into xa), or the first two (into xb)
    __device__ __forceinline__ void first(const GpLevel<T> &V, const T *b, bool two, T k1, T k2, bool one) {
        each(V.n, one, [&](int i) {
            const T ui = V.u[i], x1 = P.invtheta * ui;
            if (!two) {
                V.d[i] = sizeof(T) == 8 ? P.invtheta * b[i] : x1;
                V.xa[i] = x1;
                return;
            }
            T dg;
            const T t = gp_resid(V, i, T(0), ui, V.u, dg);  // -(A u)_i
            const T bi = b[i], r = fma(P.invtheta, t, bi);
            if constexpr (sizeof(T) == 8) {
                const T e = fma(k2, r, k1 * P.invtheta * bi);
                V.d[i] = e;
                V.xb[i] = fma(V.idg[i], e, x1);
            } else {
                const T dn = k1 * x1 + k2 * r * V.idg[i];
                V.d[i] = dn;
                V.xb[i] = x1 + dn;
            }
        });
    }

    // z = M r; ends with r . z and beta
    __device__ __forceinline__ bool vcycle() {
        const int deg = P.deg;
        bool mine = true;  // does this block work on the levels at hand?
#pragma unroll 1
        for (int l = 0; l < P.nl; l++) {
            const GpLevel<T> &V = P.lv[l];
            const bool one = l >= P.tail;
            if (one && blockIdx.x != 0) {
                mine = false;
                break;
            }
            const T *b = l == 0 ? P.r : V.b;
            if (l == P.nl - 1) {
                T *out = l == 0 ? P.z : V.xb;
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
                    first(V, b, false, T(0), T(0), one);
                    if (!step(one)) return false;
                    T *cur = V.xa;
#pragma unroll 1
                    for (int k = 1; k < 8; k++) {
                        T *o = k == 7 ? out : (cur == V.xa ? V.xb : V.xa);
                        if (o == cur) o = cur == V.xa ? V.xb : V.xa;
                        cheb<false, false>(V, b, cur, o, P.e1[k], P.e2[k], one);
                        if (!step(one)) return false;
                        cur = o;
                    }
                    if (cur != out) each(V.n, one, [&](int i) { out[i] = cur[i]; });
                }
                if (!step(one)) return false;
                break;
            }
            T *cur = deg >= 2 ? V.xb : V.xa;
            first(V, b, deg >= 2, deg >= 2 ? P.c1[1] : T(0), deg >= 2 ? P.c2[1] : T(0), one);
            if (!step(one)) return false;
#pragma unroll 1
            for (int k = 2; k < deg; k++) {
                T *o = cur == V.xa ? V.xb : V.xa;
                cheb<false, false>(V, b, cur, o, P.c1[k], P.c2[k], one);
                if (!step(one)) return false;
                cur = o;
            }
            // the residual of every row, then the members' sums of every aggregate (in member order)
            each(V.n, one, [&](int i) {
                T dg;
                V.d[i] = gp_resid(V, i, b[i], cur[i], cur, dg);
            });
            if (!step(one)) return false;
            const GpLevel<T> &W = P.lv[l + 1];
            each(W.n, one, [&](int I) {
                T a = 0;
                const int k1 = V.mrp[I + 1];
                for (int k = V.mrp[I]; k < k1; k++) a += V.d[V.mci[k]];
                W.b[I] = a;
                W.u[I] = a * W.idg[I];
            });
            // the tail's block reads what the others wrote, and they wait for its last barrier
            if (!(one ? step(true) : bar.sync())) return false;
        }
#pragma unroll 1
        for (int l = P.nl - 2; l >= 0; l--) {
            const GpLevel<T> &V = P.lv[l], &W = P.lv[l + 1];
            const bool one = l >= P.tail;
            if (one && !mine) continue;
            if (!one && l + 1 >= P.tail && !bar.sync()) return false;  // the tail is done
            const T *b = l == 0 ? P.r : V.b;
            // where pre-smoothing left its iterate
            T *cur = (deg % 2 == 0) ? V.xb : V.xa;
            each(V.n, one, [&](int i) {
                const int a = V.agg[i];
                if (a >= 0 && !V.dir[i]) cur[i] += P.scale * W.xb[a];
            });
            if (!step(one)) return false;
#pragma unroll 1
            for (int k = 0; k < deg; k++) {
                const bool last = k == deg - 1, rz = last && l == 0;
                T *o = rz ? P.z : (cur == V.xa ? V.xb : V.xa);
                if (rz) {
                    const Acc<T> a = k == 0 ? cheb<true, true>(V, b, cur, o, T(0), P.invtheta, false)
                                            : cheb<false, true>(V, b, cur, o, P.c1[k], P.c2[k], false);
                    if (!reduce<T, 1>(a, Acc<T>(), [&](double2 t) { set_beta(t.x); })) return false;
                } else {
                    if (k == 0) cheb<true, false>(V, b, cur, o, T(0), P.invtheta, one);
                    else cheb<false, false>(V, b, cur, o, P.c1[k], P.c2[k], one);
                    if (!step(one)) return false;
                }
                cur = o;
            }
        }
        if (P.nl == 1) {  // no smoothing pass: the coarsest solve's r . z
            Acc<double> a;
            each(P.lv[0].n, false, [&](int i) { a.v += (double)P.r[i] * (double)P.z[i]; });
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

    __device__ __forceinline__ void run() {
        const int n = P.lv[0].n;
        const int *rp = P.lv[0].rp, *ci = P.lv[0].ci;
        if constexpr (sizeof(T) == 8) {
            Acc<double> rr, bb;
            each(n, false, [&](int i) {
                double dg;
                const double bi = P.b64[i];
                const double ri = bi - gp_flux(rp, ci, P.v64, P.leak64, i, P.x64[i], P.x64, dg);
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
            for (int it = 0;; it++) {
                if (!vcycle()) return;
                const double beta = s.beta;
                each(n, false, [&](int i) { P.p[i] = beta == 0.0 ? P.z[i] : P.z[i] + beta * P.p[i]; });
                if (!bar.sync() || it > P.maxiter) return;
                Acc<double> a;
                each(n, false, [&](int i) {
                    double dg;
                    const double pi = P.p[i], v = gp_flux(rp, ci, P.v64, P.leak64, i, pi, P.p, dg);
                    P.q[i] = v;
                    a.v += pi * v;
                });
                if (!reduce<double, 1>(a, Acc<double>(), [&](double2 t) { set_alpha(t.x); })) return;
                if (!s.active) return;
                const double al = s.alpha;
                Acc<double> c;
                each(n, false, [&](int i) {
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
                each(n, false, [&](int i) {
                    double dg;
                    const double xi = P.x64[i], bi = P.b64[i];
                    const double ri = bi - gp_flux(rp, ci, P.v64, P.leak64, i, xi, P.x64, dg);
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
                const double inv = 1.0 / s.scale, scale = s.scale;
                each(n, false, [&](int i) {
                    const float2 v = df_from_double(P.r64[i] * inv);
                    P.rd[i] = v;
                    put_r(i, v.x);
                });
                if (!bar.sync()) return;
                for (int it = 0;; it++) {
                    if (!vcycle()) return;
                    const double beta = s.beta;
                    const float2 bd = df_from_double(beta);
                    each(n, false, [&](int i) {
                        const float2 zi = make_float2(P.z[i], 0.0f);
                        P.pd[i] = beta == 0.0 ? zi : df_add(zi, df_mul(bd, P.pd[i]));
                    });
                    if (!bar.sync()) return;
                    if (it > P.maxiter) break;
                    Acc<float> a;
                    each(n, false, [&](int i) {
                        const float2 pi = P.pd[i];
                        float2 v = df_mul(P.leakdf[i], pi);
                        const int e1 = rp[i + 1];
                        for (int e = rp[i]; e < e1; e++) v = df_add(v, df_mul(P.vdf[e], df_sub(pi, P.pd[ci[e]])));
                        P.qd[i] = v;
                        a = a + Acc<float>::prod(pi.x, v.x);
                    });
                    if (!reduce<float, 1>(a, Acc<float>(), [&](double2 t) { set_alpha(t.x); })) return;
                    if (!s.active) break;
                    const float2 al = df_from_double(s.alpha);
                    const double as = s.alpha * scale;
                    Acc<float> c;
                    each(n, false, [&](int i) {
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
    if (threadIdx.x == 0) {
        memset(&st, 0, sizeof(st));
        st.cont = 1.0;
    }
    __syncthreads();
    GpSolve<T> S{P, GridBar{P.bar, P.expired}, st, 0};
    S.run();
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) P.st[0] = st;
}

}  // namespace dpf
