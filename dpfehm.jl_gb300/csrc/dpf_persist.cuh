// dpf_persist.cuh -- a whole CG + AMG solve of a regular-grid handle as one cooperative launch.
//
// What bounds a solve of up to a few million cells is not its cells but its steps: a V-cycle is
// about five kernels per level, each some microseconds of launch, drain and last-block reduction
// however small its level (100 x 100 x 10 cells in FP64: 152 us per iteration, 17 us of them FP64
// work). Here one block per SM stays resident and the steps are separated by grid barriers (1.5 us after
// the last block arrives). The scalars of a single problem are formed by every block for itself, and
// convergence is decided on the device. The prolongation costs no step: whoever finishes a coarse cell
// adds it to its eight children. Levels of any size are spread over all SMs, which FP64 steps need (GB300
// issues 1.6 FP64 instructions per clock and SM): the fused tail of 1875 cells took 65 us on one.
//
// Measured, forward + pullback, separate kernels -> one launch: FP64 50x50x5 3.42 -> 1.80 ms, 100x100x10
// 4.57 -> 2.41 ms, 200x200x25 13.4 -> 7.2 ms, 20 grids of about 8k cells 4.41 -> 2.90 ms; mixed, 5
// transient steps of 800k cells 46.6 -> 35.9 ms, 100x100x10 2.55 -> 2.03 ms; 152 grids of 1000 cells FP64 2.97 -> 2.26 ms,
// mixed 2.04 -> 1.70 ms.
//
// Per cell the arithmetic is that of the per-level kernels (the shared cell_* functions), so both
// give the same iterates up to the order of the reductions; FP64 V-cycles of two steps take r D^-1 from
// the pass that makes r (stored in the level's direction buffer, free until the post-smoothing), one
// multiplication per cell instead of seven.
//
// Per problem and level the cells are cut into equal shares, at most one per block over the batch; a
// share's reduction has its own slot, so sums do not depend on where in a batch a problem lies.
// Registers: 80 at 768 threads, with next to no spills. Spilled values cost more here than elsewhere: a
// barrier invalidates L1, and local memory with it (out-of-line passes with 300 bytes of spills and
// stack took 222 us per iteration of 800k mixed cells against 175).
#pragma once
#include "dpf_grid.cuh"

namespace dpf {

constexpr int kPersistThreads = 768;
constexpr int kPersistTail32 = 2048, kPersistTail64 = 512;  // cells of a one-block tail's first level
constexpr int kPersistTailBytes = 80 * 1024;  // shared memory for a single problem's tail
constexpr int kPersistLevels = 16;
constexpr int kPersistProblems = 256;  // (and at most one per block)
static_assert(2 * kPersistProblems <= kPersistThreads, "two lanes per problem sum the slots");

struct PersistSegs {
    const int4 *list;    // {problem, piece, pieces of the problem, 0}
    const int2 *pinfo;   // per problem {first, count}
    int n;
};

template <typename T>
struct PersistLevel {
    const LevelDesc *desc;
    Coeffs<T> C;
    T *xa, *xb, *b, *d;
    const uint8_t *dir;
    PersistSegs smooth;  // cells of the problems smoothed on this level
    PersistSegs restr;   // cells of the next level of those problems
};

template <typename T>
struct PersistParams {
    PersistLevel<T> lv[kPersistLevels];
    int nlev, nprob, deg, onelevel;  // onelevel: some problem's finest level is its coarsest
    T c1[8], c2[8], invtheta, scale, u1;  // u1 = (1 + c1[1]) invtheta
    PersistSegs all;     // finest cells of every problem
    const int2 *tail;    // per problem {first level of its one-block tail, coarsest level}
    const double *Inv;
    CgState *st;
    int *count;
    unsigned *bar;
    int *expired;
    double2 *partials;   // two halves of nslots
    int nslots, lane_bits;  // 1 << lane_bits lanes per problem sum its slots
    double tol2;
    int maxiter, max_rounds, zero_guess, tail_bytes;
    const double *b64;
    double *x64;
    T *r, *z;            // the V-cycle's right-hand side and result
    double *p, *q;       // FP64 CG
    double *r64;         // mixed: true residual; double-float CG
    float2 *rd, *pd, *qd;
    CoeffsDF cdf;
    Coeffs<double> C64;
};

// ---- the passes of a V-cycle over cells [c0, c1) of one problem's level, by one block; the grid-wide levels
// and the one-block tail share them

// the first two Chebyshev steps from a zero guess (one, for degree 1)
template <typename T>
__device__ __forceinline__ void pass_first(const PersistParams<T> &P, const PersistLevel<T> &V, const LevelDesc &Ls,
                                        const T *b, int c0, int c1) {
    const LevelDesc L = Ls;
#pragma unroll 1
    for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
        Cell c;
        cell_at(L, li, c);
        if constexpr (sizeof(T) == 8) {
            if (P.deg == 2) {  // from u = b D^-1, stored with b
                const T *u = V.d;
                const T ui = u[c.i];
                T dg;
                const T t = resid7(L, c, V.C, [] { return T(0); }, ui, [&](long long j, int, int, int) { return u[j]; }, dg);
                const T r = fma(P.invtheta, t, b[c.i]);
                V.xb[c.i] = fma(P.c2[1] * V.C.idg[c.i], r, P.u1 * ui);
                continue;
            }
        }
        if (P.deg >= 2) cell_cheb_first2<T>(L, c, V.C, b, V.xb, V.d, P.invtheta, P.c1[1], P.c2[1]);
        else cell_cheb_first<T>(L, c, V.C, b, V.xa, V.d, P.invtheta);
    }
}

// The children of a coarse cell on the level above (V, descriptor Lf): their values are read before the
// coarse cell's own step, whose result is then added to them (read one after another, at the end, they
// took 3 us a step).
template <typename T>
struct Children {
    T v[8];
    long long i0;
    unsigned on;
    __device__ __forceinline__ void read(const PersistParams<T> &P, const PersistLevel<T> &V, const LevelDesc &Lf,
                                         const Cell &cc) {
        const T *x = (P.deg % 2 == 0) ? V.xb : V.xa;  // where pre-smoothing left its iterate
        const bool ox = 2 * cc.ix + 1 < Lf.nx, oy = 2 * cc.iy + 1 < Lf.ny, oz = 2 * cc.iz + 1 < Lf.nz;
        const long long sx = (long long)Lf.ny * Lf.nz, sy = Lf.nz;
        i0 = Lf.off + (2 * cc.ix) * sx + (2 * cc.iy) * sy + 2 * cc.iz;
        on = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const bool in = (!(k & 4) || ox) && (!(k & 2) || oy) && (!(k & 1) || oz);
            const long long i = i0 + (k & 4 ? sx : 0) + (k & 2 ? sy : 0) + (k & 1);
#if DPF_CHECKED
            if (in && !DPF_INSIDE(CK_ONE_CHILD, i, Lf.off, Lf.off + Lf.n)) {
                v[k] = T(0);
                continue;
            }
#endif
            v[k] = in ? x[i] : T(0);
            if (in && !V.dir[i]) on |= 1u << k;
        }
    }
    __device__ __forceinline__ void add(const PersistParams<T> &P, const PersistLevel<T> &V, const LevelDesc &Lf, T e) {
        T *x = (P.deg % 2 == 0) ? V.xb : V.xa;
        const long long sx = (long long)Lf.ny * Lf.nz, sy = Lf.nz;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (on >> k & 1) x[i0 + (k & 4 ? sx : 0) + (k & 2 ? sy : 0) + (k & 1)] = v[k] + P.scale * e;
    }
};

// Chebyshev step: FIRST of the post-smoothing, or with the direction of the one before. UP: it is the level's
// last, and adds its iterate to the level above; DOT: returns the sum of b . x over the thread's cells.
template <typename T, bool FIRST, bool UP, bool DOT>
__device__ __forceinline__ Acc<T> pass_step(const PersistParams<T> &P, const PersistLevel<T> &V, const LevelDesc &Ls,
                                            const T *b, const T *cur, T *o, int k, int c0, int c1,
                                            const PersistLevel<T> *up, const LevelDesc *Lfs) {
    const LevelDesc L = Ls;
    const T k1 = P.c1[k], k2 = FIRST ? P.invtheta : P.c2[k];
    Acc<T> a;
#pragma unroll 1
    for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
        Cell c;
        cell_at(L, li, c);
        Children<T> ch;
        if constexpr (UP) ch.read(P, *up, *Lfs, c);
        T bi;
        const T xo = cell_cheb_step<T, FIRST>(L, c, V.C, b, cur, o, V.d, k1, k2, bi);
        if constexpr (UP) ch.add(P, *up, *Lfs, xo);
        if constexpr (DOT) a = a + Acc<T>::prod(bi, xo);
    }
    return a;
}

// Restriction of b - A x into cells [c0, c1) of the next level W. FP32: eight lanes per coarse cell, one
// child each, summed in the children's order like the per-level kernel. FP64: four lanes with the two
// children of a z pair each (the sums between lanes are FP64 instructions too: 1.1 a child against 3).
template <typename T>
__device__ __forceinline__ void pass_restrict(const PersistParams<T> &P, const PersistLevel<T> &V,
                                           const PersistLevel<T> &W, const LevelDesc &Ls, const LevelDesc &Lcs,
                                           const T *b, const T *cur, int c0, int c1) {
    constexpr int kLanes = sizeof(T) == 8 ? 4 : 8;
    const LevelDesc L = Ls, Lc = Lcs;
    const int g = threadIdx.x & (kLanes - 1);
#pragma unroll 1
    for (int l0 = c0; l0 < c1; l0 += kPersistThreads / kLanes) {
        const int li = l0 + (int)(threadIdx.x / kLanes);
        T v = T(0);
        Cell cc;
        if (li < c1) {
            cell_at(Lc, li, cc);
            Cell c;
            c.ix = 2 * cc.ix + (sizeof(T) == 8 ? g >> 1 : g >> 2);
            c.iy = 2 * cc.iy + (sizeof(T) == 8 ? g & 1 : (g >> 1) & 1);
            c.iz = 2 * cc.iz + (sizeof(T) == 8 ? 0 : g & 1);
            if (c.ix < L.nx && c.iy < L.ny)
#pragma unroll 1
                for (int z = 0; z < (sizeof(T) == 8 ? 2 : 1); z++, c.iz++)
                    if (c.iz < L.nz) {
                        c.i = L.off + ((long long)c.ix * L.ny + c.iy) * L.nz + c.iz;
                        T dg;
                        const T r = resid7(L, c, V.C, [&] { return b[c.i]; }, cur[c.i],
                                           [&](long long j, int, int, int) { return cur[j]; }, dg);
                        v = z ? v + r : r;
                    }
        }
        T s;
        if constexpr (sizeof(T) == 8) {
            s = v + __shfl_xor_sync(0xffffffffu, v, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
        } else {
            s = T(0);
#pragma unroll
            for (int k = 0; k < 8; k++) s += __shfl_sync(0xffffffffu, v, k, 8);
        }
        if (li < c1 && g == 0) {
            W.b[cc.i] = s;
            if constexpr (sizeof(T) == 8)
                if (P.deg == 2) W.d[cc.i] = s * W.C.idg[cc.i];
        }
    }
}

// A block's share of a list: problem, cells, slot, and the descriptors of the list's level and of the
// level next to it (the level above for `smooth`, whose results go there; the finer one for `restr`).
struct Piece {
    int p, c0, c1, slot;
    LevelDesc L, M;
};

template <typename T>
struct PersistShared {
    Piece all, smooth[kPersistLevels], restr[kPersistLevels];  // p < 0: no share
    LevelDesc tail[kPersistLevels];   // of the problem whose tail this block is at
    PersistLevel<T> tl[kPersistLevels];  // a single problem's levels, the tail's arrays in shared memory
    uint8_t act[kPersistProblems];    // the problems still active
    CgState one;
    int one_count;
};

// One block's view.
template <typename T, bool kSingle>
struct Persist {
    PersistShared<T> &sh;
    const PersistParams<T> &P;
    GridBar bar;
    CgState *st;              // the problems' states; a single one's and its count in shared memory
    int *count;
    static constexpr bool single = kSingle;
    int half = 0;             // of the reduction slots, in use

    // one thread: this block's share of a list
    __device__ __forceinline__ void find(const PersistSegs &S, int level, int other, Piece &w) const {
        w.p = -1;
        if ((int)blockIdx.x >= S.n) return;
        const int4 g = single ? make_int4(0, blockIdx.x, S.n, 0) : S.list[blockIdx.x];
        w.p = g.x;
        w.slot = blockIdx.x;
        w.L = P.lv[level].desc[g.x];
        w.M = P.lv[other].desc[g.x];
        // equal shares of the groups of 32 cells, the first ones one group longer
        const int n = (int)w.L.n, units = (n + 31) >> 5, base = units / g.z, more = units - base * g.z;
        w.c0 = min(n, 32 * (g.y * base + min(g.y, more)));
        w.c1 = min(n, 32 * ((g.y + 1) * base + min(g.y + 1, more)));
    }
    // f(share) for a share of an active problem
    template <typename F>
    __device__ __forceinline__ void share(const Piece &w, F f) const {
        if (w.p >= 0 && (single || sh.act[w.p])) f(w);
    }
    // the block's sum of one or two accumulators to a piece's slot
    template <typename A, int NV>
    __device__ __forceinline__ void put_sum(Acc<A> a, Acc<A> b, int slot) {
        const double2 t = block_sum<A, NV>(a, b);
        if (threadIdx.x == 0) slots()[slot] = t;
        __syncthreads();  // block_sum's shared slots are free again
    }
    // The barrier behind a phase of sums: f(problem, state, total). One problem: every block adds the slots
    // up itself, in the same order, and keeps the problem's state in shared memory (2.8 us less than
    // waiting for one block to do it); several: 2 to 32 lanes per problem in the last block to arrive, so that all
    // problems are summed at once (a warp per problem took 3.7 us for every 24 problems, four times an iteration).
    template <typename F>
    __device__ __forceinline__ bool reduce(const PersistSegs &S, F f, bool any = true) {
        if (!any) return bar.sync();
        if (!single) return bar.sync([&] { totals(S, f); });
        if (!bar.sync()) return false;
        if (threadIdx.x < 32) total_of_one(S, f);
        // the next sums go to the other half: a slower block may still be reading this one
        half ^= 1;
        __syncthreads();
        return true;
    }
    __device__ __forceinline__ double2 *slots() const { return P.partials + (half ? P.nslots : 0); }
    // one problem, by one warp (as a loop over problems: without it 1M FP64 cells took 0.8 % more, by its registers)
    template <typename F>
    __device__ __forceinline__ void total_of_one(const PersistSegs &S, F f) const {
        const int lane = threadIdx.x & 31;
#pragma unroll 1
        for (int p = (int)(threadIdx.x >> 5); p < P.nprob; p++) {
            const int2 g = single ? make_int2(0, S.n) : S.pinfo[p];
            if (g.y == 0) continue;
            double2 t = make_double2(0.0, 0.0);
#pragma unroll 1
            for (int k = lane; k < g.y; k += 32) {
                const double2 v = __ldcg(slots() + g.x + k);
                t.x += v.x;
                t.y += v.y;
            }
            t.x = warp_sum(t.x);
            t.y = warp_sum(t.y);
            if (lane == 0) f(p, st[p], t);
        }
    }
    // several problems, 1 << lane_bits lanes each
    template <typename F>
    __device__ __forceinline__ void totals(const PersistSegs &S, F f) const {
        const int lg = P.lane_bits, p = (int)threadIdx.x >> lg, q = threadIdx.x & ((1 << lg) - 1);
        // a warp without a problem has no sums to make (its FP64 additions would hold up the others')
        if ((int)(threadIdx.x & ~31u) >> lg >= P.nprob) return;
        const int2 g = p < P.nprob ? S.pinfo[p] : make_int2(0, 0);
        double2 t = make_double2(0.0, 0.0);
#pragma unroll 1
        for (int k = q; k < g.y; k += 1 << lg) {
            const double2 v = __ldcg(slots() + g.x + k);
            t.x += v.x;
            t.y += v.y;
        }
#pragma unroll
        for (int l = 4; l >= 0; l--)
            if (l < lg) {
                t.x += __shfl_xor_sync(0xffffffffu, t.x, 1 << l);
                t.y += __shfl_xor_sync(0xffffffffu, t.y, 1 << l);
            }
        if (q == 0 && g.y > 0) f(p, st[p], t);
    }
    template <typename V>
    __device__ __forceinline__ V scalar(const V *v) const {
        return single ? *v : __ldcg(v);
    }
    // b_i of a finest row and, FP64 with the two-step start, r_i / a_ii for the first smoothing pass
    __device__ __forceinline__ void put_r(long long i, T r) const {
        P.r[i] = r;
        if constexpr (sizeof(T) == 8)
            if (P.deg == 2 && P.nlev > 1) P.lv[0].d[i] = r * P.lv[0].C.idg[i];
    }
    __device__ __forceinline__ const T *rhs(int l) const { return l == 0 ? P.r : P.lv[l].b; }

    // post-smoothing step k of a level below the finest
    __device__ __forceinline__ void step_any(const PersistLevel<T> &V, const LevelDesc &L, const T *b, const T *cur, T *o,
                                             int k, int c0, int c1, const PersistLevel<T> *up, const LevelDesc *Lf) {
        if (k < P.deg - 1) {
            if (k == 0) pass_step<T, true, false, false>(P, V, L, b, cur, o, k, c0, c1, up, Lf);
            else pass_step<T, false, false, false>(P, V, L, b, cur, o, k, c0, c1, up, Lf);
        } else {
            if (k == 0) pass_step<T, true, true, false>(P, V, L, b, cur, o, k, c0, c1, up, Lf);
            else pass_step<T, false, true, false>(P, V, L, b, cur, o, k, c0, c1, up, Lf);
        }
    }
    __device__ __forceinline__ const PersistLevel<T> &level(int l) const {
        if constexpr (single) return sh.tl[l];
        else return P.lv[l];
    }
    // A single problem: the tail's arrays in its block's shared memory, coarsest level first, while they fit;
    // what other blocks write of its first level stays where it is. A tail's steps wait for the trips of
    // their loads and stores: five steps of 800k mixed cells 34.6 -> 33.9 ms, 100k mixed cells 1.94 -> 1.84 ms,
    // 12k FP64 cells 1.76 -> 1.73 ms.
    __device__ __forceinline__ void stage_tail(unsigned char *mem) {
        using CT = coef_t<T>;
        if ((int)threadIdx.x < P.nlev) sh.tl[threadIdx.x] = P.lv[threadIdx.x];
        const int2 g = P.tail[0];
        int used = 0;
#pragma unroll 1
        for (int l = g.y; l >= max(g.x, 1); l--) {
            __syncthreads();
            const PersistLevel<T> &V = P.lv[l];
            const long long off = sh.tail[l].off;
            const int n = (int)sh.tail[l].n;
            const bool dense = l == g.y, mine_b = l > g.x, mine_d = l > g.x || sizeof(T) == 4;
            constexpr int kPlain = sizeof(T) == 8 ? 2 : 1;  // idg, dg
            const int need = (n * (dense ? (int)sizeof(T) : (int)sizeof(T) * (4 + kPlain) + 4 * (int)sizeof(CT) + 1) + 15) & ~15;
            if (used + need > P.tail_bytes) continue;
            T *t = (T *)(mem + used);
            used += need;
            if (dense) {
                if (mine_b && threadIdx.x == 0) sh.tl[l].b = t - off;
                continue;
            }
            T *idg = t + 4 * n, *dg = idg + n;
            CT *c = (CT *)(t + (4 + kPlain) * n);
            uint8_t *dir = (uint8_t *)(c + 4 * n);
            for (int k = threadIdx.x; k < n; k += kPersistThreads) {
                idg[k] = V.C.idg[off + k];
                if constexpr (sizeof(T) == 8) dg[k] = V.C.dg[off + k];
                c[k] = V.C.cx[off + k];
                c[n + k] = V.C.cy[off + k];
                c[2 * n + k] = V.C.cz[off + k];
                c[3 * n + k] = V.C.leak[off + k];
                dir[k] = V.dir[off + k];
            }
            if (threadIdx.x == 0) {
                PersistLevel<T> &W = sh.tl[l];
                W.xa = t - off;
                W.xb = t + n - off;
                if (mine_b) W.b = t + 2 * n - off;
                if (mine_d) W.d = t + 3 * n - off;
                W.C.idg = idg - off;
                if constexpr (sizeof(T) == 8) W.C.dg = dg - off;
                W.C.cx = c - off;
                W.C.cy = c + n - off;
                W.C.cz = c + 2 * n - off;
                W.C.leak = c + 3 * n - off;
                W.dir = dir - off;
            }
        }
        __syncthreads();
    }
    // the small levels of problem p and the dense coarsest solve, by this block
    __device__ __forceinline__ void tail(int p, int lt, int lc) {
        const LevelDesc *L, *M;
        T *cur = nullptr;
        if (!single) {  // a single problem's were read at the start
            __syncthreads();
            if ((int)threadIdx.x >= lt - 1 && (int)threadIdx.x <= lc) sh.tail[threadIdx.x] = P.lv[threadIdx.x].desc[p];
            __syncthreads();
        }
#pragma unroll 1
        for (int l = lt; l < lc; l++) {
            const PersistLevel<T> &V = level(l);
            L = &sh.tail[l];
            M = &sh.tail[l + 1];
            pass_first(P, V, *L, V.b, 0, (int)L->n);
            cur = P.deg >= 2 ? V.xb : V.xa;
            __syncthreads();
#pragma unroll 1
            for (int k = 2; k < P.deg; k++) {
                T *o = cur == V.xa ? V.xb : V.xa;
                pass_step<T, false, false, false>(P, V, *L, V.b, cur, o, k, 0, (int)L->n, nullptr, nullptr);
                cur = o;
                __syncthreads();
            }
            pass_restrict(P, V, level(l + 1), *L, *M, V.b, cur, 0, (int)M->n);
            __syncthreads();
        }
        {
            // eight lanes per row: a row's products in one chain took longer than a level's smoothing
            const PersistLevel<T> &V = level(lc);
            L = &sh.tail[lc];
            M = &sh.tail[lc - 1];
            const int n = (int)L->n, i = threadIdx.x >> 3, s = threadIdx.x & 7;
            const double *Ip = P.Inv + (long long)p * kMaxCoarse * kMaxCoarse;
            if (threadIdx.x < 8 * kMaxCoarse) {
                double x = 0.0;
                if (i < n)
#pragma unroll 4
                    for (int j = s; j < n; j += 8) x = fma(Ip[j * kMaxCoarse + i], (double)V.b[L->off + j], x);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                if (i < n && s == 0) {
                    Cell c;
                    cell_at(*L, i, c);
                    Children<T> ch;
                    ch.read(P, level(lc - 1), *M, c);
                    ch.add(P, level(lc - 1), *M, (T)x);
                }
            }
            __syncthreads();
        }
#pragma unroll 1
        for (int l = lc - 1; l >= lt; l--) {
            const PersistLevel<T> &V = level(l);
            L = &sh.tail[l];
            M = &sh.tail[l - 1];
            cur = (P.deg % 2 == 0) ? V.xb : V.xa;
#pragma unroll 1
            for (int k = 0; k < P.deg; k++) {
                T *o = cur == V.xa ? V.xb : V.xa;
                step_any(V, *L, V.b, cur, o, k, 0, (int)L->n, &level(l - 1), M);
                cur = o;
                __syncthreads();
            }
        }
    }

    // z = M r; the finest level's last pass also sums r . z and sets beta
    __device__ __forceinline__ bool vcycle() {
        const int deg = P.deg;
#pragma unroll 1
        for (int l = 0; l + 1 < P.nlev; l++) {
            const PersistLevel<T> &V = P.lv[l];
            if (V.smooth.n == 0) continue;
            const T *b = rhs(l);
            T *cur = deg >= 2 ? V.xb : V.xa;
            share(sh.smooth[l], [&](const Piece &w) { pass_first(P, V, w.L, b, w.c0, w.c1); });
            if (!bar.sync()) return false;
#pragma unroll 1
            for (int k = 2; k < deg; k++) {
                T *o = cur == V.xa ? V.xb : V.xa;
                share(sh.smooth[l], [&](const Piece &w) {
                    pass_step<T, false, false, false>(P, V, w.L, b, cur, o, k, w.c0, w.c1, nullptr, nullptr);
                });
                cur = o;
                if (!bar.sync()) return false;
            }
            share(sh.restr[l], [&](const Piece &w) {
                pass_restrict(P, V, P.lv[l + 1], w.M, w.L, b, cur, w.c0, w.c1);
            });
            if (!bar.sync()) return false;
        }
#pragma unroll 1
        for (int p = blockIdx.x; p < P.nprob; p += gridDim.x) {
            if (!single && !sh.act[p]) continue;
            const int2 g = P.tail[p];
            if (g.x > 0) {
                tail(p, g.x, g.y);
                continue;
            }
            // a problem of one level: z = A^-1 r and r . z
            const LevelDesc L = P.lv[0].desc[p];
            const int n = (int)L.n, i = threadIdx.x;
            const double *Ip = P.Inv + (long long)p * kMaxCoarse * kMaxCoarse;
            double x = 0.0;
            if (i < n)
#pragma unroll 1
                for (int j = 0; j < n; j++) x += Ip[j * kMaxCoarse + i] * (double)P.r[L.off + j];
            if (i < n) P.z[L.off + i] = (T)x;
            Acc<double> a;
            if (i < n) a.v = (double)P.r[L.off + i] * (double)(T)x;
            const double2 t = block_sum<double, 1>(a, Acc<double>());
            const int2 g0 = single ? make_int2(0, P.all.n) : P.all.pinfo[p];
            for (int k = threadIdx.x; k < g0.y; k += kPersistThreads)
                slots()[g0.x + k] = k == 0 ? t : make_double2(0.0, 0.0);
            __syncthreads();
        }
        if (!reduce(P.all, [&](int p, CgState &s, double2 t) {
                if (s.active && P.tail[p].x == 0) set_beta(s, t.x);
            }, P.onelevel != 0))
            return false;
        // post-smoothing; the last pass of a level adds its iterate to the level above
#pragma unroll 1
        for (int l = P.nlev - 2; l >= 0; l--) {
            const PersistLevel<T> &V = P.lv[l];
            if (V.smooth.n == 0) continue;
            const T *b = rhs(l);
            T *cur = (deg % 2 == 0) ? V.xb : V.xa;
#pragma unroll 1
            for (int k = 0; k < deg; k++) {
                const bool last = k == deg - 1, rz = last && l == 0;
                T *o = rz ? P.z : (cur == V.xa ? V.xb : V.xa);
                share(sh.smooth[l], [&](const Piece &w) {
                    if (!rz) {
                        step_any(V, w.L, b, cur, o, k, w.c0, w.c1, &P.lv[l > 0 ? l - 1 : 0], &w.M);
                        return;
                    }
                    const Acc<T> a =
                        k == 0 ? pass_step<T, true, false, true>(P, V, w.L, b, cur, o, k, w.c0, w.c1, nullptr, nullptr)
                               : pass_step<T, false, false, true>(P, V, w.L, b, cur, o, k, w.c0, w.c1, nullptr, nullptr);
                    put_sum<T, 1>(a, Acc<T>(), w.slot);
                });
                cur = o;
                if (!reduce(V.smooth, [&](int, CgState &s, double2 t) {
                        if (s.active) set_beta(s, t.x);
                    }, rz))
                    return false;
            }
        }
        return true;
    }
    __device__ __forceinline__ static void set_beta(CgState &s, double rz) {
        s.rz_old = s.rz;
        s.rz = rz;
        s.beta = (s.iters == 0 || s.rz_old == 0.0) ? 0.0 : s.rz / s.rz_old * s.cont;
        s.cont = 1.0;
    }
};

// The solve. T = double: FP64 CG; T = float: rounds of double-float CG with an FP32 V-cycle, each started
// from and checked against the true FP64 residual.
template <typename T, bool kSingle>
__device__ __forceinline__ void persist_solve(Persist<T, kSingle> &S) {
    const PersistParams<T> &P = S.P;
    int *const count = S.count;
    // after a reduction: which problems go on, and whether any does
    auto refresh = [&](bool round) {
        if (!S.single)
            for (int p = threadIdx.x; p < P.nprob; p += kPersistThreads)
                S.sh.act[p] = round ? __ldcg(&S.st[p].ru_flag) != 0 : __ldcg(&S.st[p].active) != 0;
        const int n = S.single ? *count : __ldcg(count);
        __syncthreads();
        return n > 0;
    };
    auto fresh_state = [&](CgState &s) {
        memset(&s, 0, sizeof(s));
        s.cont = 1.0;
        s.tol2 = P.tol2;
        s.status = DPF_OK;
    };
    auto end_iteration = [&](CgState &s, double rr, bool met, int iters) {
        s.rr = rr;
        s.iters++;
        s.total_iters++;
        if (!isfinite(s.rr)) {
            s.status = DPF_NAN;
            deactivate(s, count);
        } else if (met) {
            deactivate(s, count);
        } else if (iters + 1 >= P.maxiter) {
            s.status = DPF_NOT_CONVERGED;
            deactivate(s, count);
        }
    };

    if constexpr (sizeof(T) == 8) {
        const Coeffs<double> C = P.lv[0].C;
        const double *bv = P.b64;
        double *x = P.x64;
        // r = b - A x
        S.share(S.sh.all, [&](const Piece &w) {
            const LevelDesc L = w.L;
            const int c0 = w.c0, c1 = w.c1, slot = w.slot;
            Acc<double> rr, bb;
#pragma unroll 1
            for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                Cell c;
                cell_at(L, li, c);
                double Ax, dg;
                apply7(L, c, C, x[c.i], [&](long long j, int, int, int) { return x[j]; }, Ax, dg);
                const double bi = bv[c.i], ri = bi - Ax;
                S.put_r(c.i, ri);
                rr.v += ri * ri;
                if (!P.lv[0].dir[c.i]) bb.v += bi * bi;
            }
            S.template put_sum<double, 2>(rr, bb, slot);
        });
        if (!S.reduce(P.all, [&](int, CgState &s, double2 t) {
                fresh_state(s);
                s.rr = t.x;
                s.bb = t.y;
                bool go = s.bb > 0.0 && s.rr > P.tol2 * s.bb;
                if (!isfinite(s.rr)) {
                    s.status = DPF_NAN;
                    go = false;
                }
                s.active = go ? 1 : 0;
                if (go) atomicAdd(count, 1);
            }))
            return;
        if (!refresh(false)) return;
        for (int it = 0;; it++) {
            if (!S.vcycle()) return;
            S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc &L = w.L;
                const int p = w.p, c0 = w.c0, c1 = w.c1;
                const double beta = S.scalar(&S.st[p].beta);
#pragma unroll 2
                for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                    const long long i = L.off + li;
                    P.p[i] = beta == 0.0 ? P.z[i] : P.z[i] + beta * P.p[i];
                }
            });
            if (!S.bar.sync() || it >= P.maxiter + 1) return;
            S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc L = w.L;
                const int c0 = w.c0, c1 = w.c1, slot = w.slot;
                Acc<double> a;
#pragma unroll 1
                for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                    Cell c;
                    cell_at(L, li, c);
                    const double pi = P.p[c.i];
                    double Ax, dg;
                    apply7(L, c, C, pi, [&](long long j, int, int, int) { return P.p[j]; }, Ax, dg);
                    P.q[c.i] = Ax;
                    a.v += pi * Ax;
                }
                S.template put_sum<double, 1>(a, Acc<double>(), slot);
            });
            if (!S.reduce(P.all, [&](int, CgState &s, double2 t) {
                    if (s.active) finish_pq(s, t.x, count);
                }))
                return;
            S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc L = w.L;
                const int p = w.p, c0 = w.c0, c1 = w.c1, slot = w.slot;
                if (!S.scalar(&S.st[p].active)) return;
                const double al = S.scalar(&S.st[p].alpha);
                Acc<double> a;
#pragma unroll 2
                for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                    const long long i = L.off + li;
                    const double xi = x[i], pi = P.p[i], r0 = P.r[i], qi = P.q[i];
                    x[i] = xi + al * pi;
                    const double ri = r0 - al * qi;
                    S.put_r(i, ri);
                    a.v += ri * ri;
                }
                S.template put_sum<double, 1>(a, Acc<double>(), slot);
            });
            if (!S.reduce(P.all, [&](int, CgState &s, double2 t) {
                    if (s.active) end_iteration(s, t.x, t.x <= s.tol2 * s.bb, s.iters);
                }))
                return;
            if (!refresh(false)) return;
        }
    } else {
        for (int round = -1; round < P.max_rounds; round++) {
            // the true residual: before the first round, and after each
            const bool first = round < 0;
            S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc L = w.L;
                const int c0 = w.c0, c1 = w.c1, slot = w.slot;
                Acc<double> rr, bb;
#pragma unroll 1
                for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                    Cell c;
                    const uint8_t id = P.lv[0].dir[L.off + li];
                    double ri, xi = 0.0;
                    float dg = 0.0f;
                    const double bi = P.b64[L.off + li];
                    if (first && P.zero_guess) {
                        c.i = L.off + li;
                        ri = id ? 0.0 : bi;
                    } else {
                        cell_at(L, li, c);
                        xi = P.x64[c.i];
                        double Ax;
                        apply7_f32diag(L, c, P.C64, P.lv[0].C, xi, P.x64, Ax, dg);
                        ri = bi - Ax;
                    }
                    P.r64[c.i] = ri;
                    rr.v += ri * ri;
                    if (id) continue;
                    if (first) {
                        bb.v += bi * bi;
                    } else {
                        const double f = (double)fmaf(2.0f * dg, abs_float_trunc(xi), abs_float_trunc(bi));
                        bb.v = fma(f, f, bb.v);
                    }
                }
                if (!first) bb.v *= 0x1p-96;
                S.template put_sum<double, 2>(rr, bb, slot);
            });
            // (every problem still counted as active has left the round: only a pass cap can end it early)
            if (!S.reduce(P.all, [&](int, CgState &s, double2 t) {
                    if (!first && !s.ru_flag) return;
                    if (first) fresh_state(s);
                    deactivate(s, count);
                    check_round(s, first, t, P.tol2, P.maxiter, P.max_rounds, count);
                }))
                return;
            if (!refresh(true) || round + 1 >= P.max_rounds) return;
            // r = r64 / scale
            S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc &L = w.L;
                const int p = w.p, c0 = w.c0, c1 = w.c1;
                const double inv = 1.0 / S.scalar(&S.st[p].scale);
                for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                    const long long i = L.off + li;
                    const double w = P.r64[i] * inv;
                    float2 v;
                    double w48;
                    if (!split48(w, v.x, v.y, w48)) v = df_from_double(w);
                    P.rd[i] = v;
                    P.r[i] = v.x;
                }
            });
            if (!S.bar.sync()) return;
            for (int it = 0;; it++) {
                if (!S.vcycle()) return;
                S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc &L = w.L;
                const int p = w.p, c0 = w.c0, c1 = w.c1;
                    const double beta = S.scalar(&S.st[p].beta);
                    const float2 bd = df_from_double(beta);
#pragma unroll 2
                    for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                        const long long i = L.off + li;
                        const float2 zi = make_float2(P.z[i], 0.0f);
                        P.pd[i] = beta == 0.0 ? zi : df_add(zi, df_mul(bd, P.pd[i]));
                    }
                });
                if (!S.bar.sync()) return;
                if (it >= P.maxiter + 1) break;
                S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc L = w.L;
                const int c0 = w.c0, c1 = w.c1, slot = w.slot;
                    Acc<float> a;
#pragma unroll 1
                    for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                        Cell c;
                        cell_at(L, li, c);
                        const float2 pi = P.pd[c.i];
                        const float2 v = cell_df_apply(L, c, P.cdf, pi, P.pd);
                        P.qd[c.i] = v;
                        a = a + Acc<float>::prod(pi.x, v.x);
                    }
                    S.template put_sum<float, 1>(a, Acc<float>(), slot);
                });
                if (!S.reduce(P.all, [&](int, CgState &s, double2 t) {
                        if (s.active) finish_pq(s, t.x, count);
                    }))
                    return;
                S.share(S.sh.all, [&](const Piece &w) {
                const LevelDesc L = w.L;
                const int p = w.p, c0 = w.c0, c1 = w.c1, slot = w.slot;
                    if (!S.scalar(&S.st[p].active)) return;
                    const double alpha = S.scalar(&S.st[p].alpha), as = alpha * S.scalar(&S.st[p].scale);
                    const float2 al = df_from_double(alpha);
                    Acc<float> a;
#pragma unroll 2
                    for (int li = c0 + (int)threadIdx.x; li < c1; li += kPersistThreads) {
                        const long long i = L.off + li;
                        const float2 pi = P.pd[i];
                        P.x64[i] = fma(as, (double)pi.x + (double)pi.y, P.x64[i]);
                        const float2 ri = df_sub(P.rd[i], df_mul(al, P.qd[i]));
                        P.rd[i] = ri;
                        P.r[i] = ri.x;
                        a = a + Acc<float>::prod(ri.x, ri.x);
                    }
                    S.template put_sum<float, 1>(a, Acc<float>(), slot);
                });
                if (!S.reduce(P.all, [&](int, CgState &s, double2 t) {
                        if (s.active)
                            end_iteration(s, t.x, t.x * s.scale * s.scale <= s.tol2 * s.obb || t.x <= kRoundDrop2,
                                          s.total_iters);
                    }))
                    return;
                if (!refresh(false)) break;
            }
            refresh(true);  // the problems of this round, for its check
        }
    }
}

// kSingle: a handle of one problem
template <typename T, bool kSingle>
__global__ void __launch_bounds__(kPersistThreads, 1) k_solve_persistent(const __grid_constant__ PersistParams<T> P) {
    __shared__ PersistShared<T> sh;
    constexpr bool single = kSingle;
    for (int p = threadIdx.x; p < P.nprob; p += kPersistThreads) sh.act[p] = 1;
    if (threadIdx.x == 0) {
        sh.one_count = 0;
        memset(&sh.one, 0, sizeof(sh.one));
    }
    __syncthreads();
    Persist<T, kSingle> S{sh, P, GridBar{P.bar, P.expired}, single ? &sh.one : P.st,
                          single ? &sh.one_count : P.count};
    {
        const int l = threadIdx.x & 31, what = threadIdx.x >> 5;
        if (what == 0 && l < P.nlev) S.find(P.lv[l].smooth, l, max(l - 1, 0), sh.smooth[l]);
        if (what == 1 && l + 1 < P.nlev) S.find(P.lv[l].restr, l + 1, l, sh.restr[l]);
        if (what == 2 && l == 0) S.find(P.all, 0, 0, sh.all);
        if (what == 3 && l < P.nlev && single) sh.tail[l] = P.lv[l].desc[0];
    }
    __syncthreads();
    if constexpr (single) {
        extern __shared__ __align__(16) unsigned char persist_mem[];
        if (blockIdx.x == 0 && P.tail[0].x > 0) S.stage_tail(persist_mem);
    }
    persist_solve(S);
    __syncthreads();
    if (single && blockIdx.x == 0 && threadIdx.x == 0) {
        P.st[0] = sh.one;
        *P.count = sh.one_count;
    }
}

}  // namespace dpf
