// dpf_front.cu -- nested dissection, fronts, and their factorisation and solves (see dpf_front.h).
//
// What bounds it: GB300 issues about two FP64 multiply-adds per clock and SM, so every kernel here
// is FP64-issue- or latency-bound, never by memory. Tiles are therefore small (32 x 32), to spread
// the few fronts near the root over all SMs.
#include "dpf_front.h"

#include <algorithm>
#include <cmath>
#include <mutex>
#include <set>
#include <stdexcept>
#include <string>

#include "dpf_struct.h"
#include "dpf_means.cuh"

namespace dpf {

namespace {

constexpr int kLeaf = 16;          // cells of a leaf at most
constexpr int kNB = 16;            // own columns of one step of a large front
constexpr int kTile = 32;          // tile edge of the large fronts
constexpr int kSmallM = 76;        // fronts of at most this many rows factor in one block's shared memory
constexpr int kSmallThreads = 128;
constexpr int kStepThreads = 256;
constexpr int kSolveThreads = 256;
constexpr int kSolveRows = 32;     // rows of a forward block
constexpr int kStepBuf = kNB * kNB + kNB;  // Z_TT and the pivots, behind a front's L columns

int blocks_of(int n, int b) { return (n + b - 1) / b; }

// ------------------------------------------------------------------ small fronts: one block each
// The whole front in shared memory (column-major, odd leading dimension): its panel with the
// operator's entries, the children's update matrices added in order, then per own column c a
// Gauss-Jordan step: with the multipliers l_i = S_ic / S_cc, the trailing columns lose l_i S_jc
// and the finished ones (which hold Z and -W) l_i S_cj; column c becomes (1, -l). Results: the
// panel, the update matrix (lower part) and 1 / pivot. The trailing triangle's columns are paired,
// the longest with the shortest, so that a step's elements form two full rectangles and no lane of an
// FP64 instruction is idle: fronts of 21 rows would otherwise use a third of each (225 us for the
// 16142 leaves of a 500 x 500 grid with a warp per column).
__global__ void __launch_bounds__(kSmallThreads)
k_front_small(const int *__restrict__ list, const Front *__restrict__ fr, const int *__restrict__ child,
              const int *__restrict__ rel, double *__restrict__ panels, const double *__restrict__ pool_in,
              double *__restrict__ pool_out, double *__restrict__ dinv, int *err) {
    extern __shared__ double sm[];
    const Front f = fr[list[blockIdx.x]];
    const int m = f.m, k = f.k, u = m - k, ld = m | 1;
    double *S = sm, *lv = sm + (size_t)ld * m, *cv = lv + m;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, nth = (int)blockDim.x, nw = nth >> 5;
    double *P = panels + f.panel;
    for (int j = w; j < m; j += nw)
        for (int i = lane; i < m; i += 32) S[j * ld + i] = j < k ? P[(size_t)j * m + i] : 0.0;
    __syncthreads();
    for (int q = 0; q < f.nch; q++) {
        const Front c = fr[child[f.ch0 + q]];
        const int cu = c.m - c.k;
        const double *U = pool_in + c.upd;
        const int *R = rel + c.rows;
        for (int j = w; j < cu; j += nw) {
            const int pj = R[j];
            for (int i = j + lane; i < cu; i += 32) S[pj * ld + R[i]] += U[(size_t)j * cu + i];
        }
        __syncthreads();  // children add to the same entries one after another
    }
    for (int c = 0; c < k; c++) {
        if (w == 0) {
            double p = S[c * ld + c];
            if (!(p > 0.0)) {  // not positive definite: recorded; a unit pivot keeps the rest finite
                if (lane == 0) atomicExch(err, 1);
                p = 1.0;
            }
            const double rp = recip(p);
            if (lane == 0) dinv[f.first + c] = rp;
            for (int i = c + 1 + lane; i < m; i += 32) {
                const double v = S[c * ld + i];
                cv[i] = v;
                lv[i] = -v * rp;
            }
        }
        __syncthreads();
        const int h = m - c - 1;          // rows below the pivot
        const int len = h + 1;            // of a pair of trailing columns: h - p and p + 1 rows
        const int npair = (h + 1) >> 1;   // pair p: columns c + 1 + p and c + 1 + (h - 1 - p)
        const int ntri = npair * len, nall = ntri + h * c;
        const float rlen = 1.0f / (float)len, rh = 1.0f / (float)(h > 0 ? h : 1);
        for (int x = t; x < nall; x += nth) {
            int i, j;
            double a;
            if (x < ntri) {
                int p = (int)(((float)x + 0.5f) * rlen), e = x - p * len;
                const int top = h - p;    // rows of the pair's longer column
                const int p2 = h - 1 - p;
                if (e < top) {
                    j = c + 1 + p;
                    i = j + e;
                } else {
                    if (p2 <= p) continue;  // the middle column of an odd count has no partner
                    j = c + 1 + p2;
                    i = j + (e - top);
                }
                a = cv[j];
            } else {
                const int y = x - ntri;
                j = (int)(((float)y + 0.5f) * rh);
                i = c + 1 + (y - j * h);
                a = S[j * ld + c];
            }
            S[j * ld + i] = fma(lv[i], a, S[j * ld + i]);
        }
        for (int i = c + t; i < m; i += nth) S[c * ld + i] = i == c ? 1.0 : lv[i];
        __syncthreads();
    }
    for (int j = w; j < k; j += nw)
        for (int i = lane; i < m; i += 32) P[(size_t)j * m + i] = i >= j ? S[j * ld + i] : 0.0;
    double *O = pool_out + f.upd;
    for (int j = w; j < u; j += nw)
        for (int i = j + lane; i < u; i += 32) O[(size_t)j * u + i] = S[(k + j) * ld + k + i];
}

// ------------------------------------------------------------------ large fronts
// add the update matrix of child number q into the parent's panel and update matrix (one launch
// per child: two children of a front reach the same entries, and their order stays fixed)
__global__ void __launch_bounds__(kStepThreads)
k_front_extend(const int *__restrict__ list, const Front *__restrict__ fr, const int *__restrict__ child,
               const int *__restrict__ rel, double *__restrict__ panels, const double *__restrict__ pool_in,
               double *__restrict__ pool_out, int q) {
    const Front f = fr[list[blockIdx.y]];
    if (q >= f.nch) return;
    const Front c = fr[child[f.ch0 + q]];
    const int cu = c.m - c.k, u = f.m - f.k;
    const int nt = (cu + kTile - 1) / kTile;
    if (nt == 0) return;
    const int ti = (int)blockIdx.x / nt, tj = (int)blockIdx.x - ti * nt;
    if (ti >= nt || tj > ti) return;
    const double *U = pool_in + c.upd;
    const int *R = rel + c.rows;
    const int i = ti * kTile + (threadIdx.x & 31);
    if (i >= cu) return;
    const int pi = R[i];
    for (int jj = threadIdx.x >> 5; jj < kTile; jj += kStepThreads / 32) {
        const int j = tj * kTile + jj;
        if (j >= cu || j > i) continue;
        const int pj = R[j];
        double *dst = pj < f.k ? panels + f.panel + (size_t)pj * f.m + pi
                               : pool_out + f.upd + (size_t)(pj - f.k) * u + (pi - f.k);
        *dst += U[(size_t)j * cu + i];
    }
}

// Step s, first half, on the own columns T = [16 s, 16 s + jb): every block eliminates the 16 x 16
// diagonal block in shared memory (Gauss-Jordan: Z_TT and the pivots, one element per thread, the same
// arithmetic in every block), then makes one piece: block 0 stores Z_TT and the pivots, the
// next ones 32 rows of the multipliers below T, L_iT = F_iT Z_TT^T D^-1 (to the step buffer), the
// rest 32 finished columns of the rows T, Z_Tj = Z_TT R_Tj (in place).
// 16 columns: the chain over a step's pivots is bound by FP64 latency (about 550 clocks a column), and
// separators of 7, 15, 31 ... cells fill them; with 32 columns a step took 44 us here and 17 us in
// the update, whatever the front, and fronts of 15 own columns did twice their work.
__global__ void __launch_bounds__(kStepThreads)
k_front_panel(const int *__restrict__ list, const Front *__restrict__ fr, double *__restrict__ panels,
              double *__restrict__ lbuf, double *__restrict__ dinv, int s, int *err) {
    const Front f = fr[list[blockIdx.y]];
    const int m = f.m, t0 = s * kNB;
    if (t0 >= f.k) return;
    const int jb = min(kNB, f.k - t0), below = m - t0 - jb;
    const int nr = (below + kTile - 1) / kTile, nc = (t0 + kTile - 1) / kTile;
    const int piece = (int)blockIdx.x - 1;  // -1: the diagonal block; then nr row pieces, nc column pieces
    if (piece >= nr + nc) return;
    __shared__ double D[kNB][kNB + 1];      // D[j][i]: column j, row i
    __shared__ double A[kTile][kTile + 1];
    __shared__ double lv[kNB], cv[kNB], pv[kNB], rv[kNB];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    constexpr int kWarps = kStepThreads / 32;
    double *P = panels + f.panel;
    const int r0 = t0 + jb + piece * kTile, c0 = (piece - nr) * kTile;
    const int rn = min(kTile, m - r0), cn = min(kTile, t0 - c0);
    const int di = t & 15, dj = t >> 4;
    static_assert(kStepThreads == kNB * kNB && kNB == 16, "one element of the diagonal block per thread");
    D[dj][di] = (di < jb && dj < jb) ? (di >= dj ? P[(size_t)(t0 + dj) * m + t0 + di] : 0.0) : (di == dj ? 1.0 : 0.0);
    if (piece >= nr) {
        // A[e][j]: row e of T, column c0 + j
        for (int j = w * 2 + (lane >> 4); j < kTile; j += 2 * kWarps)
            A[lane & 15][j] = (j < cn && (lane & 15) < jb) ? P[(size_t)(c0 + j) * m + t0 + (lane & 15)] : 0.0;
    } else if (piece >= 0) {
        for (int e = w; e < kNB; e += kWarps)  // A[e][i]: column e of T, row r0 + i
            A[e][lane] = (lane < rn && e < jb) ? P[(size_t)(t0 + e) * m + r0 + lane] : 0.0;
    }
    __syncthreads();
    for (int c = 0; c < jb; c++) {
        if (w == 0) {
            double p = D[c][c];
            if (!(p > 0.0)) {
                if (lane == 0 && piece < 0) atomicExch(err, 1);
                p = 1.0;
            }
            const double rp = recip(p);
            if (lane < kNB) {
                const double v = D[c][lane];
                cv[lane] = v;
                lv[lane] = lane > c ? -v * rp : 0.0;
            }
            if (lane == 0) {
                pv[c] = p;
                rv[c] = rp;
            }
        }
        __syncthreads();
        if (dj == c) {
            if (di >= c) D[c][di] = di == c ? 1.0 : lv[di];
        } else if (di > c && (dj < c || di >= dj)) {
            D[dj][di] = fma(lv[di], dj < c ? D[dj][c] : cv[dj], D[dj][di]);
        }
        __syncthreads();
    }
    double *Lb = lbuf + f.lbuf;
    if (piece < 0) {
        double *X = Lb + (size_t)kNB * m;
        X[dj * kNB + di] = di >= dj ? D[dj][di] : 0.0;
        if (t < jb) {
            X[kNB * kNB + t] = pv[t];
            dinv[f.first + t0 + t] = rv[t];
        }
    } else if (piece < nr) {
        // thread: row lane, columns w and w + 8
        for (int c = w; c < jb; c += kWarps) {
            double v = 0.0;
            for (int e = 0; e <= c; e++) v = fma(A[e][lane], D[e][c], v);
            if (lane < rn) Lb[(size_t)c * m + r0 + lane] = v * rv[c];
        }
    } else {
        // thread: rows w and w + 8 of T, column lane
        for (int r = w; r < jb; r += kWarps) {
            double v = 0.0;
            for (int e = 0; e <= r; e++) v = fma(D[e][r], A[e][lane], v);
            if (lane < cn) P[(size_t)(c0 + lane) * m + t0 + r] = v;
        }
    }
}

// Step s, second half: C_ij -= L_iT B_j^T for the rows i below T; B_j = L_jT D for the columns behind
// T (own ones or the update matrix, j <= i), Z_Tj^T for the finished ones, Z_TT^T for T itself
// (whose C starts at zero). Tiles of 32 x 32 from the first row below T and from column 0; the
// first block also stores Z_TT in the panel.
__global__ void __launch_bounds__(kStepThreads)
k_front_update(const int *__restrict__ list, const Front *__restrict__ fr, double *__restrict__ panels,
               double *__restrict__ pool, const double *__restrict__ lbuf, int s, int ncol) {
    const Front f = fr[list[blockIdx.y]];
    const int m = f.m, u = m - f.k, t0 = s * kNB;
    if (t0 >= f.k) return;
    const int jb = min(kNB, f.k - t0), t1 = t0 + jb;
    const int ti = (int)blockIdx.x / ncol, tj = (int)blockIdx.x - ti * ncol;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    constexpr int kWarps = kStepThreads / 32;
    double *P = panels + f.panel;
    const double *Lb = lbuf + f.lbuf, *X = Lb + (size_t)kNB * m, *pv = X + kNB * kNB;
    if (blockIdx.x == 0 && t < kNB * kNB) {
        const int i = t & 15, j = t >> 4;
        if (i < jb && j < jb) P[(size_t)(t0 + j) * m + t0 + i] = X[j * kNB + i];
    }
    const int i0 = t1 + ti * kTile, j0 = tj * kTile;
    const int in = min(kTile, m - i0), jn = min(kTile, m - j0);
    if (in <= 0 || jn <= 0 || j0 > i0 + in - 1) return;
    __shared__ double A[kNB][kTile + 1];  // A[c][i] = -L_i,c
    __shared__ double B[kNB][kTile + 1];  // B[c][j]
    for (int c = w; c < kNB; c += kWarps) {
        A[c][lane] = (c < jb && lane < in) ? -Lb[(size_t)c * m + i0 + lane] : 0.0;
        const int j = j0 + lane;
        if (j >= t1) B[c][lane] = (c < jb && j < m) ? Lb[(size_t)c * m + j] * pv[c] : 0.0;
    }
    if (j0 < t1)  // a row of T per half warp's lane: consecutive in the panel
        for (int jj = w * 2 + (lane >> 4); jj < kTile; jj += 2 * kWarps) {
            const int j = j0 + jj, c = lane & 15;
            if (j < t0) B[c][jj] = c < jb ? P[(size_t)j * m + t0 + c] : 0.0;
            else if (j < t1) B[c][jj] = X[(j - t0) * kNB + c];
        }
    __syncthreads();
    // thread: row lane, columns w, w + 8, w + 16, w + 24
    double v[4];
    double *C[4];
    const int i = i0 + lane;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int jj = w + q * kWarps, j = j0 + jj;
        const bool ok = lane < in && jj < jn && j <= i;
        C[q] = !ok ? nullptr : j < f.k ? P + (size_t)j * m + i : pool + f.upd + (size_t)(j - f.k) * u + (i - f.k);
        v[q] = ok && (j < t0 || j >= t1) ? *C[q] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < kNB; c++) {
        const double a = A[c][lane];
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = fma(a, B[c][w + q * kWarps], v[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (C[q]) *C[q] = v[q];
}

// ------------------------------------------------------------------ solves
// Forward, one tree level: t = (right-hand side of the own cells, 0) + the children's update vectors
// (every block of a front builds it in shared memory, the children in order), then 32 rows of
// G t1 per block, eight warps sharing the own columns: D^-1 Z t1 to y, t2 - W t1 to the front's
// update vector.
__global__ void __launch_bounds__(kSolveThreads)
k_front_fwd(const int *__restrict__ list, const Front *__restrict__ fr, const int *__restrict__ child,
            const int *__restrict__ rel, const double *__restrict__ panels, const double *__restrict__ dinv,
            const double *__restrict__ b, double *__restrict__ y, double *__restrict__ vec) {
    extern __shared__ double sm[];
    const Front f = fr[list[blockIdx.y]];
    const int m = f.m, k = f.k, r0 = (int)blockIdx.x * kSolveRows;
    if (r0 >= m) return;
    __shared__ double red[kSolveThreads / 32][kSolveRows + 1];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    constexpr int kWarps = kSolveThreads / 32;
    for (int i = t; i < m; i += kSolveThreads) sm[i] = i < k ? b[f.first + i] : 0.0;
    __syncthreads();
    for (int q = 0; q < f.nch; q++) {
        const Front c = fr[child[f.ch0 + q]];
        const int cu = c.m - c.k;
        const int *R = rel + c.rows;
        for (int e = t; e < cu; e += kSolveThreads) sm[R[e]] += vec[c.vec + e];
        __syncthreads();
    }
    const int i = r0 + lane;
    double v = 0.0;
    if (i < m) {
        const double *G = panels + f.panel + i;
        const int ce = min(k, i + 1);
#pragma unroll 8
        for (int c = w; c < ce; c += kWarps) v = fma(G[(size_t)c * m], sm[c], v);
    }
    red[w][lane] = v;
    __syncthreads();
    if (w == 0 && i < m) {
        double s = red[0][lane];
#pragma unroll
        for (int q = 1; q < kWarps; q++) s += red[q][lane];
        if (i < k) y[f.first + i] = s * dinv[f.first + i];
        else vec[f.vec + (i - k)] = sm[i] + s;
    }
}

// Backward, one tree level: x1 = G^T (D^-1 y, x2), cols own columns per block, a warp per column.
__global__ void __launch_bounds__(kSolveThreads)
k_front_bwd(const int *__restrict__ list, const Front *__restrict__ fr, const int *__restrict__ rows,
            const double *__restrict__ panels, const double *__restrict__ y, double *__restrict__ x, int cols) {
    extern __shared__ double sm[];
    const Front f = fr[list[blockIdx.y]];
    const int m = f.m, k = f.k, c0 = (int)blockIdx.x * cols;
    if (c0 >= k) return;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    constexpr int kWarps = kSolveThreads / 32;
    for (int i = t; i < m; i += kSolveThreads) sm[i] = i < k ? y[f.first + i] : x[rows[f.rows + i - k]];
    __syncthreads();
    const int ce = min(k, c0 + cols);
    for (int c = c0 + w; c < ce; c += kWarps) {
        const double *G = panels + f.panel + (size_t)c * m;
        double v = 0.0;
#pragma unroll 8
        for (int i = c + lane; i < m; i += 32) v = fma(G[i], sm[i], v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) x[f.first + c] = v;
    }
}

// The same for the small fronts, a warp per front (four in a block): a leaf's block of 256 threads
// would hold more idle warps than rows (44 and 62 us for the leaves of a 500 x 500 grid).
constexpr int kWarpFronts = 4;
__global__ void __launch_bounds__(32 * kWarpFronts)
k_front_fwd_warp(const int *__restrict__ list, int count, const Front *__restrict__ fr, const int *__restrict__ child,
                 const int *__restrict__ rel, const double *__restrict__ panels, const double *__restrict__ dinv,
                 const double *__restrict__ b, double *__restrict__ y, double *__restrict__ vec) {
    __shared__ double sh[kWarpFronts][kSmallM + 1];
    const int lane = threadIdx.x & 31, at = (int)blockIdx.x * kWarpFronts + (int)(threadIdx.x >> 5);
    if (at >= count) return;
    double *sm = sh[threadIdx.x >> 5];
    const Front f = fr[list[at]];
    const int m = f.m, k = f.k;
    for (int i = lane; i < m; i += 32) sm[i] = i < k ? b[f.first + i] : 0.0;
    __syncwarp();
    for (int q = 0; q < f.nch; q++) {
        const Front c = fr[child[f.ch0 + q]];
        const int cu = c.m - c.k;
        const int *R = rel + c.rows;
        for (int e = lane; e < cu; e += 32) sm[R[e]] += vec[c.vec + e];
        __syncwarp();
    }
    for (int i = lane; i < m; i += 32) {
        const double *G = panels + f.panel + i;
        const int ce = min(k, i + 1);
        double v = 0.0;
#pragma unroll 4
        for (int c = 0; c < ce; c++) v = fma(G[(size_t)c * m], sm[c], v);
        if (i < k) y[f.first + i] = v * dinv[f.first + i];
        else vec[f.vec + (i - k)] = sm[i] + v;
    }
}
// a lane per own column here: the sums need no exchange between lanes
__global__ void __launch_bounds__(32 * kWarpFronts)
k_front_bwd_warp(const int *__restrict__ list, int count, const Front *__restrict__ fr, const int *__restrict__ rows,
                 const double *__restrict__ panels, const double *__restrict__ y, double *__restrict__ x) {
    __shared__ double sh[kWarpFronts][kSmallM + 1];
    const int lane = threadIdx.x & 31, at = (int)blockIdx.x * kWarpFronts + (int)(threadIdx.x >> 5);
    if (at >= count) return;
    double *sm = sh[threadIdx.x >> 5];
    const Front f = fr[list[at]];
    const int m = f.m, k = f.k;
    for (int i = lane; i < m; i += 32) sm[i] = i < k ? y[f.first + i] : x[rows[f.rows + i - k]];
    __syncwarp();
    for (int c = lane; c < k; c += 32) {
        const double *G = panels + f.panel + (size_t)c * m;
        double v = 0.0;
#pragma unroll 4
        for (int i = c; i < m; i++) v = fma(G[i], sm[i], v);
        x[f.first + c] = v;
    }
}

__global__ void k_front_gather(int n, const int *__restrict__ perm, const double *__restrict__ b,
                               double *__restrict__ y) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = b[perm[i]];
}
__global__ void k_front_scatter(int n, const int *__restrict__ perm, const double *__restrict__ y,
                                double *__restrict__ x) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[perm[i]] = y[i];
}

__global__ void k_direct_resid(int n, const uint8_t *__restrict__ dir, const double *__restrict__ b,
                               const double *__restrict__ Ax, double *acc) {
    double rr = 0.0, bb = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (dir[i]) continue;
        const double r = b[i] - Ax[i];
        rr = fma(r, r, rr);
        bb = fma(b[i], b[i], bb);
    }
    for (int o = 16; o > 0; o >>= 1) {
        rr += __shfl_xor_sync(0xffffffffu, rr, o);
        bb += __shfl_xor_sync(0xffffffffu, bb, o);
    }
    __shared__ double sr[8], sb[8];
    if ((threadIdx.x & 31) == 0) {
        sr[threadIdx.x >> 5] = rr;
        sb[threadIdx.x >> 5] = bb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) {
            rr += sr[w];
            bb += sb[w];
        }
        atomicAdd(&acc[0], rr);
        atomicAdd(&acc[1], bb);
    }
}

void fck(cudaError_t e, const char *what) {
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw CudaError(std::string("direct solve, ") + what + ": " + cudaGetErrorString(e), e);
    }
}

}  // namespace

// ================================================================== ordering
namespace {
// nodes in an order with children before parents; returns the node's number
struct Builder {
    Dissection d;
    int add(const std::vector<int> &cells, int depth, const std::vector<int> &children) {
        const int id = (int)d.k.size();
        d.first.push_back((int)d.perm.size());
        d.k.push_back((int)cells.size());
        d.parent.push_back(-1);
        d.depth.push_back(depth);
        d.perm.insert(d.perm.end(), cells.begin(), cells.end());
        for (int c : children) d.parent[c] = id;
        return id;
    }
};

// the box [lo, hi) of a grid with strides st, offset off: halved across its longest axis
int dissect_box(Builder &B, std::array<int, 3> lo, std::array<int, 3> hi, const long long st[3], long long off,
                int depth) {
    const int e[3] = {hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]};
    const long long cells = (long long)e[0] * e[1] * e[2];
    if (cells <= 0) return -1;
    std::vector<int> own, ch;
    auto take = [&](std::array<int, 3> a, std::array<int, 3> b) {
        for (int x = a[0]; x < b[0]; x++)
            for (int y = a[1]; y < b[1]; y++)
                for (int z = a[2]; z < b[2]; z++) own.push_back((int)(off + x * st[0] + y * st[1] + z * st[2]));
    };
    if (cells <= kLeaf) {
        take(lo, hi);
        return B.add(own, depth, ch);
    }
    int ax = 0;
    for (int k = 1; k < 3; k++)
        if (e[k] > e[ax]) ax = k;
    const int mid = lo[ax] + e[ax] / 2;
    auto h1 = hi, l2 = lo, sl = lo, sh = hi;
    h1[ax] = mid;
    l2[ax] = mid + 1;
    sl[ax] = mid;
    sh[ax] = mid + 1;
    for (int c : {dissect_box(B, lo, h1, st, off, depth + 1), dissect_box(B, l2, hi, st, off, depth + 1)})
        if (c >= 0) ch.push_back(c);
    take(sl, sh);
    return B.add(own, depth, ch);
}

// A set of a graph's vertices (those with tag[v] == id): its connected components packed into two
// halves when there are several, otherwise cut by one level of a breadth-first search from a
// pseudo-peripheral vertex (George and Liu's automatic nested dissection): the smallest level that
// leaves at least 30 % of the vertices on either side, without the vertices that touch no later level.
struct GraphCut {
    const std::vector<int> &rp, &ci;
    Builder &B;
    std::vector<int> tag, level;
    int next_tag = 0;
    GraphCut(const std::vector<int> &rp_, const std::vector<int> &ci_, Builder &B_, int n)
        : rp(rp_), ci(ci_), B(B_), tag(n, -1), level(n, -1) {}

    // breadth-first search from s within tag id: vertices in order, level[] set (the caller resets it)
    void bfs(int s, int id, std::vector<int> &out) {
        out.clear();
        out.push_back(s);
        level[s] = 0;
        for (size_t h = 0; h < out.size(); h++)
            for (int e = rp[out[h]]; e < rp[out[h] + 1]; e++) {
                const int v = ci[e];
                if (tag[v] == id && level[v] < 0) {
                    level[v] = level[out[h]] + 1;
                    out.push_back(v);
                }
            }
    }
    int cut(std::vector<int> set, int depth) {
        if (set.empty()) return -1;
        if ((int)set.size() <= kLeaf) return B.add(set, depth, {});
        const int id = next_tag++;
        for (int v : set) tag[v] = id;
        std::vector<std::vector<int>> comps;
        std::vector<int> order;
        for (int v : set)
            if (level[v] < 0) {
                bfs(v, id, order);
                comps.push_back(order);
            }
        for (int v : set) level[v] = -1;
        std::vector<int> left, right, sep, ch;
        if (comps.size() > 1) {
            std::stable_sort(comps.begin(), comps.end(),
                             [](const std::vector<int> &a, const std::vector<int> &b) { return a.size() > b.size(); });
            for (auto &c : comps) {
                auto &to = left.size() <= right.size() ? left : right;
                to.insert(to.end(), c.begin(), c.end());
            }
        } else {
            // pseudo-peripheral start: twice the last vertex reached
            int s = comps[0].back();
            for (int k = 0; k < 2; k++) {
                bfs(s, id, order);
                for (int v : order) level[v] = -1;
                s = order.back();
            }
            bfs(s, id, order);
            const int nl = level[order.back()] + 1;
            std::vector<int> size(nl, 0);
            for (int v : order) size[level[v]]++;
            int best = -1;
            const double n = (double)order.size();
            double before = 0;
            for (int l = 0; l < nl; l++) {
                const double after = n - before - size[l];
                if (before >= 0.3 * n && after >= 0.3 * n && (best < 0 || size[l] < size[best])) best = l;
                before += size[l];
            }
            if (best < 0) {  // levels too thick to balance: the one that holds the median vertex
                before = 0;
                for (int l = 0; l < nl && best < 0; l++) {
                    before += size[l];
                    if (before >= 0.5 * n) best = l;
                }
            }
            for (int v : order) {
                if (level[v] < best) left.push_back(v);
                else if (level[v] > best) right.push_back(v);
                else {
                    bool touches = false;
                    for (int e = rp[v]; e < rp[v + 1] && !touches; e++)
                        touches = tag[ci[e]] == id && level[ci[e]] == best + 1;
                    (touches ? sep : left).push_back(v);
                }
            }
            for (int v : order) level[v] = -1;
            if (left.empty() || right.empty()) {  // nothing to halve: one dense node
                std::vector<int> all(order);
                return B.add(all, depth, {});
            }
        }
        std::vector<int>().swap(set);
        comps.clear();
        comps.shrink_to_fit();
        for (auto *half : {&left, &right}) {
            const int c = cut(std::move(*half), depth + 1);
            if (c >= 0) ch.push_back(c);
        }
        return B.add(sep, depth, ch);
    }
};
}  // namespace

Dissection dissect_regular(const std::vector<std::array<int, 3>> &dims, const std::vector<long long> &off) {
    Builder B;
    for (size_t p = 0; p < dims.size(); p++) {
        const long long st[3] = {(long long)dims[p][1] * dims[p][2], dims[p][2], 1};
        dissect_box(B, {0, 0, 0}, dims[p], st, off[p], 0);
    }
    return B.d;
}

Dissection dissect_graph(int n, const std::vector<int> &rp, const std::vector<int> &ci) {
    Builder B;
    GraphCut G(rp, ci, B, n);
    std::vector<int> all(n);
    for (int i = 0; i < n; i++) all[i] = i;
    G.cut(std::move(all), 0);
    return B.d;
}

Dissection dissect_band(const BandOrder &o) {
    Builder B;
    const int n = (int)o.perm.size(), nodes = blocks_of(n, kBandBlock);
    for (int s = 0; s < nodes; s++) {
        const int a = s * kBandBlock, b = std::min(n, a + kBandBlock);
        B.add(std::vector<int>(o.perm.begin() + a, o.perm.begin() + b), nodes - 1 - s,
              s ? std::vector<int>{s - 1} : std::vector<int>{});
    }
    return B.d;
}

void regular_graph(const std::vector<std::array<int, 3>> &dims, const std::vector<long long> &off,
                   std::vector<int> &rp, std::vector<int> &ci) {
    long long n = 0;
    for (size_t p = 0; p < dims.size(); p++) n = std::max(n, off[p] + (long long)dims[p][0] * dims[p][1] * dims[p][2]);
    rp.assign(1, 0);
    rp.reserve(n + 1);
    ci.clear();
    ci.reserve(6 * n);
    for (size_t p = 0; p < dims.size(); p++) {
        const int nx = dims[p][0], ny = dims[p][1], nz = dims[p][2];
        const int sx = ny * nz, sy = nz;
        int i = (int)off[p];
        for (int x = 0; x < nx; x++)
            for (int y = 0; y < ny; y++)
                for (int z = 0; z < nz; z++, i++) {
                    if (x > 0) ci.push_back(i - sx);
                    if (y > 0) ci.push_back(i - sy);
                    if (z > 0) ci.push_back(i - 1);
                    if (z + 1 < nz) ci.push_back(i + 1);
                    if (y + 1 < ny) ci.push_back(i + sy);
                    if (x + 1 < nx) ci.push_back(i + sx);
                    rp.push_back((int)ci.size());
                }
    }
}

double FrontTree::bytes() const {
    return 8.0 * ((double)panel_size + vec_size + pool_size[0] + pool_size[1] + lbuf_size) +
           8.0 * (double)rows.size() + 100.0 * (double)fr.size() + 40.0 * (double)node_of.size();
}

bool build_fronts(const Dissection &d, const std::vector<int> &rp, const std::vector<int> &ci, double max_bytes,
                  FrontTree &t) {
    const int n = (int)d.perm.size(), nn = (int)d.k.size();
    std::vector<int> inv(n), mark(n, -1), pos(n), nch(nn, 0);
    for (int i = 0; i < n; i++) inv[d.perm[i]] = i;
    t = FrontTree();
    t.fr.resize(nn);
    t.node_of.resize(n);
    t.depth = d.depth;
    for (int s = 0; s < nn; s++) {
        t.max_depth = std::max(t.max_depth, d.depth[s]);
        if (d.parent[s] >= 0) nch[d.parent[s]]++;
    }
    int total = 0;
    for (int s = 0; s < nn; s++) {
        t.fr[s].ch0 = total;
        t.fr[s].nch = 0;
        total += nch[s];
    }
    t.child.resize(total);
    for (int s = 0; s < nn; s++)
        if (d.parent[s] >= 0) {
            Front &p = t.fr[d.parent[s]];
            t.child[p.ch0 + p.nch++] = s;
        }
    const int nlev = t.max_depth + 1;
    std::vector<long long> pool(nlev, 0), lbuf(nlev, 0);
    std::vector<int> rows;
    for (int s = 0; s < nn; s++) {
        Front &f = t.fr[s];
        f.first = d.first[s];
        f.k = d.k[s];
        f.pad = 0;
        const int end = f.first + f.k;  // own cells and everything eliminated before them
        rows.clear();
        for (int i = f.first; i < end; i++) {
            t.node_of[i] = s;
            const int v = d.perm[i];
            for (int e = rp[v]; e < rp[v + 1]; e++) {
                const int r = inv[ci[e]];
                if (r >= end && mark[r] != s) {
                    mark[r] = s;
                    rows.push_back(r);
                }
            }
        }
        for (int q = 0; q < f.nch; q++) {
            const Front &c = t.fr[t.child[f.ch0 + q]];
            for (int e = 0; e < c.m - c.k; e++) {
                const int r = t.rows[c.rows + e];
                if (r >= end && mark[r] != s) {
                    mark[r] = s;
                    rows.push_back(r);
                }
            }
        }
        std::sort(rows.begin(), rows.end());
        const int u = (int)rows.size();
        f.m = f.k + u;
        for (int e = 0; e < u; e++) pos[rows[e]] = f.k + e;
        f.rows = (long long)t.rows.size();
        t.rows.insert(t.rows.end(), rows.begin(), rows.end());
        t.rel.resize(t.rows.size(), 0);
        for (int q = 0; q < f.nch; q++) {
            const Front &c = t.fr[t.child[f.ch0 + q]];
            for (int e = 0; e < c.m - c.k; e++) {
                const int r = t.rows[c.rows + e];
                t.rel[c.rows + e] = r < end ? r - f.first : pos[r];
            }
        }
        f.panel = t.panel_size;
        t.panel_size += (long long)f.m * f.k;
        f.vec = t.vec_size;
        t.vec_size += u;
        pool[d.depth[s]] += (long long)u * u;
        f.lbuf = 0;
        f.upd = 0;
        if (f.m > kSmallM) {
            f.lbuf = lbuf[d.depth[s]];
            lbuf[d.depth[s]] += (long long)f.m * kNB + kStepBuf;
        }
        t.max_m = std::max(t.max_m, f.m);
        t.fma += 0.5 * f.k * (double)f.m * f.m + 0.5 * (double)f.k * f.k * f.m;
        if (8.0 * ((double)t.panel_size + pool[d.depth[s]]) > max_bytes) return false;
    }
    // update matrices: a level's in the pool of its parity, the large fronts' first (zeroed together)
    std::vector<long long> at(nlev, 0);
    for (int pass = 0; pass < 2; pass++)
        for (int s = 0; s < nn; s++) {
            Front &f = t.fr[s];
            if ((f.m > kSmallM) != (pass == 0)) continue;
            f.upd = at[d.depth[s]];
            at[d.depth[s]] += (long long)(f.m - f.k) * (f.m - f.k);
        }
    for (int l = 0; l < nlev; l++) {
        t.pool_size[l & 1] = std::max(t.pool_size[l & 1], at[l]);
        t.lbuf_size = std::max(t.lbuf_size, lbuf[l]);
    }
    return t.bytes() <= max_bytes;
}

// ================================================================== solver
void configure_front_kernels() {
    static std::mutex mu;
    static std::set<int> done;
    int dev = 0;
    fck(cudaGetDevice(&dev), "device");
    std::lock_guard<std::mutex> lk(mu);
    if (done.count(dev)) return;
    int optin = 0;
    fck(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "attribute");
    for (const void *k : {(const void *)k_front_fwd, (const void *)k_front_bwd}) {
        cudaFuncAttributes a;
        fck(cudaFuncGetAttributes(&a, k), "attribute");
        fck(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)a.sharedSizeBytes),
            "attribute");
    }
    done.insert(dev);
}

FrontSolver::FrontSolver(const Dissection &d, const FrontTree &t, cudaStream_t s) : stream(s) {
    n = (int)d.perm.size();
    max_depth = t.max_depth;
    panel_size = t.panel_size;
    // per level: the small fronts, then the large ones
    std::vector<int> list;
    lv.resize(max_depth + 1);
    std::vector<std::vector<int>> small(max_depth + 1), large(max_depth + 1);
    for (int i = 0; i < (int)t.fr.size(); i++) (t.fr[i].m > kSmallM ? large : small)[t.depth[i]].push_back(i);
    for (int l = 0; l <= max_depth; l++) {
        Level &L = lv[l];
        L.small0 = (int)list.size();
        L.nsmall = (int)small[l].size();
        list.insert(list.end(), small[l].begin(), small[l].end());
        L.large0 = (int)list.size();
        L.nlarge = (int)large[l].size();
        list.insert(list.end(), large[l].begin(), large[l].end());
        for (int i : small[l]) L.max_small_m = std::max(L.max_small_m, t.fr[i].m);
        for (int i : large[l]) {
            const Front &f = t.fr[i];
            L.max_large_m = std::max(L.max_large_m, f.m);
            L.max_large_k = std::max(L.max_large_k, f.k);
            L.max_large_nch = std::max(L.max_large_nch, f.nch);
            L.upd_large = std::max(L.upd_large, f.upd + (long long)(f.m - f.k) * (f.m - f.k));
            for (int q = 0; q < f.nch; q++) {
                const Front &c = t.fr[t.child[f.ch0 + q]];
                L.max_child_u = std::max(L.max_child_u, c.m - c.k);
            }
        }
    }
    std::vector<int> iperm(n);
    for (int i = 0; i < n; i++) iperm[d.perm[i]] = i;
    auto alloc = [&](size_t bytes) {
        void *p = nullptr;
        if (dev_malloc(&p, std::max<size_t>(bytes, 16)) != cudaSuccess) {
            cudaGetLastError();
            throw OomError("direct solve: cudaMalloc of " + std::to_string(bytes) + " bytes failed");
        }
        owned.push_back(p);
        return p;
    };
    auto upload = [&](const void *src, size_t bytes) {
        void *p = alloc(bytes);
        if (bytes) fck(cudaMemcpyAsync(p, src, bytes, cudaMemcpyHostToDevice, stream), "upload");
        return p;
    };
    try {
        d_fr = (Front *)upload(t.fr.data(), t.fr.size() * sizeof(Front));
        d_child = (int *)upload(t.child.data(), t.child.size() * sizeof(int));
        d_rows = (int *)upload(t.rows.data(), t.rows.size() * sizeof(int));
        d_rel = (int *)upload(t.rel.data(), t.rel.size() * sizeof(int));
        d_node_of = (int *)upload(t.node_of.data(), t.node_of.size() * sizeof(int));
        d_list = (int *)upload(list.data(), list.size() * sizeof(int));
        d_perm = (int *)upload(d.perm.data(), n * sizeof(int));
        d_iperm = (int *)upload(iperm.data(), n * sizeof(int));
        d_panels = (double *)alloc(t.panel_size * sizeof(double));
        for (int k = 0; k < 2; k++) d_pool[k] = (double *)alloc(t.pool_size[k] * sizeof(double));
        d_vec = (double *)alloc(t.vec_size * sizeof(double));
        d_lbuf = (double *)alloc(t.lbuf_size * sizeof(double));
        d_dinv = (double *)alloc((size_t)n * sizeof(double));
        d_y = (double *)alloc((size_t)n * sizeof(double));
        d_x = (double *)alloc((size_t)n * sizeof(double));
        d_acc = (double *)alloc(2 * sizeof(double));
        d_err = (int *)alloc(sizeof(int));
        fck(cudaStreamSynchronize(stream), "upload");  // the host vectors go out of scope
    } catch (...) {
        for (void *p : owned) dev_free(p);
        throw;
    }
}

bool choose_fronts(Dissection &d, const BandOrder &band, const std::vector<int> &rp, const std::vector<int> &ci,
                   size_t free_bytes, FrontTree &t) {
    if (build_fronts(d, rp, ci, 0.5 * (double)free_bytes, t) && t.max_m <= FrontSolver::kMaxM) return true;
    d = dissect_band(band);
    return build_fronts(d, rp, ci, 0.9 * (double)free_bytes, t) && t.max_m <= FrontSolver::kMaxM;
}

std::unique_ptr<FrontSolver> make_fronts(Dissection d, const BandOrder &band, const std::vector<int> &rp,
                                         const std::vector<int> &ci, size_t free_bytes, cudaStream_t stream) {
    FrontTree t;
    if (!choose_fronts(d, band, rp, ci, free_bytes, t)) return nullptr;
    return std::unique_ptr<FrontSolver>(new FrontSolver(d, t, stream));
}

FrontSolver::~FrontSolver() {
    cudaStreamSynchronize(stream);
    for (void *p : owned) dev_free(p);
}

void FrontSolver::clear() {
    fck(cudaMemsetAsync(d_panels, 0, (size_t)panel_size * sizeof(double), stream), "clear");
}

bool FrontSolver::factor() {
    NvtxRange range("multifrontal factorisation");
    fck(cudaMemsetAsync(d_err, 0, sizeof(int), stream), "factor");
    for (int l = max_depth; l >= 0; l--) {
        const Level &L = lv[l];
        double *in = d_pool[(l + 1) & 1], *out = d_pool[l & 1];
        if (L.nsmall) {
            // a warp's worth of threads for the leaves, more where a front's columns are longer
            const int m = L.max_small_m, threads = m <= 24 ? 32 : m <= 40 ? 64 : kSmallThreads;
            const size_t smem = ((size_t)(m | 1) * m + 2 * (size_t)m) * sizeof(double);
            k_front_small<<<L.nsmall, threads, smem, stream>>>(d_list + L.small0, d_fr, d_child, d_rel, d_panels, in,
                                                              out, d_dinv, d_err);
            launches++;
        }
        if (!L.nlarge) continue;
        const int *list = d_list + L.large0;
        if (L.upd_large) fck(cudaMemsetAsync(out, 0, (size_t)L.upd_large * sizeof(double), stream), "factor");
        const int ct = blocks_of(L.max_child_u, kTile);
        // large fronts in runs that fit the grid's y dimension
        for (int a = 0; a < L.nlarge; a += 65535) {
            const int cnt = std::min(65535, L.nlarge - a);
            for (int q = 0; q < L.max_large_nch && ct > 0; q++) {
                k_front_extend<<<dim3(ct * ct, cnt), kStepThreads, 0, stream>>>(list + a, d_fr, d_child, d_rel, d_panels,
                                                                               in, out, q);
                launches++;
            }
            const int M = L.max_large_m;
            for (int s = 0; s < blocks_of(L.max_large_k, kNB); s++) {
                // rows below the step (a front's last step may be narrower: counted from its first
                // column plus one) and columns before it
                const int t0 = s * kNB, nr = blocks_of(std::max(M - t0 - 1, 1), kTile), nc = blocks_of(t0, kTile);
                const int ncol = blocks_of(M, kTile);
                k_front_panel<<<dim3(1 + nr + nc, cnt), kStepThreads, 0, stream>>>(list + a, d_fr, d_panels, d_lbuf,
                                                                                  d_dinv, s, d_err);
                k_front_update<<<dim3(nr * ncol, cnt), kStepThreads, 0, stream>>>(list + a, d_fr, d_panels, out, d_lbuf,
                                                                                 s, ncol);
                launches += 2;
            }
        }
    }
    fck(cudaGetLastError(), "factor launch");
    int h_err = 0;
    fck(cudaMemcpyAsync(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, stream), "factor");
    fck(cudaStreamSynchronize(stream), "factor");
    return h_err == 0;
}

void FrontSolver::solve(const double *b, double *x) {
    NvtxRange range("multifrontal solves");
    const unsigned g = (unsigned)std::min((n + 255) / 256, 4096);
    k_front_gather<<<g, 256, 0, stream>>>(n, d_perm, b, d_x);
    launches++;
    // d_x holds the permuted right-hand side; the backward sweep replaces it from the root down
    for (int l = max_depth; l >= 0; l--) {
        const Level &L = lv[l];
        if (L.nsmall) {
            k_front_fwd_warp<<<blocks_of(L.nsmall, kWarpFronts), 32 * kWarpFronts, 0, stream>>>(
                d_list + L.small0, L.nsmall, d_fr, d_child, d_rel, d_panels, d_dinv, d_x, d_y, d_vec);
            launches++;
        }
        for (int a = 0; a < L.nlarge; a += 65535) {
            const int here = std::min(65535, L.nlarge - a);
            k_front_fwd<<<dim3(blocks_of(L.max_large_m, kSolveRows), here), kSolveThreads,
                          L.max_large_m * sizeof(double), stream>>>(d_list + L.large0 + a, d_fr, d_child, d_rel, d_panels,
                                                                    d_dinv, d_x, d_y, d_vec);
            launches++;
        }
    }
    for (int l = 0; l <= max_depth; l++) {
        const Level &L = lv[l];
        if (L.nsmall) {
            k_front_bwd_warp<<<blocks_of(L.nsmall, kWarpFronts), 32 * kWarpFronts, 0, stream>>>(
                d_list + L.small0, L.nsmall, d_fr, d_rows, d_panels, d_y, d_x);
            launches++;
        }
        for (int a = 0; a < L.nlarge && L.max_large_k > 0; a += 65535) {
            const int here = std::min(65535, L.nlarge - a);
            // one column per warp where the level's few fronts would leave SMs idle
            const int cols = (long long)here * blocks_of(L.max_large_k, 32) >= 600 ? 32 : 8;
            k_front_bwd<<<dim3(blocks_of(L.max_large_k, cols), here), kSolveThreads, L.max_large_m * sizeof(double),
                          stream>>>(d_list + L.large0 + a, d_fr, d_rows, d_panels, d_y, d_x, cols);
            launches++;
        }
    }
    k_front_scatter<<<g, 256, 0, stream>>>(n, d_perm, d_x, x);
    launches++;
    fck(cudaGetLastError(), "solve launch");
}

double FrontSolver::relres(const uint8_t *dir, const double *b, const double *Ax) {
    fck(cudaMemsetAsync(d_acc, 0, 2 * sizeof(double), stream), "residual");
    k_direct_resid<<<(unsigned)std::min((n + 255) / 256, 1024), 256, 0, stream>>>(n, dir, b, Ax, d_acc);
    launches++;
    fck(cudaGetLastError(), "residual launch");
    double h[2] = {0.0, 0.0};
    fck(cudaMemcpyAsync(h, d_acc, sizeof(h), cudaMemcpyDeviceToHost, stream), "residual");
    fck(cudaStreamSynchronize(stream), "residual");
    return h[1] > 0 ? std::sqrt(h[0] / h[1]) : 0.0;
}

}  // namespace dpf
