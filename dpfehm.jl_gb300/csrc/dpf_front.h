// dpf_front.h -- nested-dissection multifrontal factorisation of the FP64 groundwater operator,
// the direct solver behind `linear_solver = cholesky_solver` (src/groundwater.jl:56-60).
//
// The cells are ordered by nested dissection (George 1973): a separator splits the cells in two
// halves without couplings between them, recursively, and is eliminated after both. Every tree
// node (separator or leaf) has a dense front over its own k cells and the u cells of its ancestors
// that its subtree touches (m = k + u). A 500 x 500 grid takes about 2e9 multiply-adds this way
// against 3e10 in its band, and, more important on a GPU, the fronts of one tree level are
// independent: the factorisation runs level by level (about log2(n / 16) of them) instead of in
// n / 32 dependent block steps, and so do the triangular solves.
//
// Per front the elimination is Gauss-Jordan on the own columns: besides the pivots d it leaves the
// m x k panel G = [Z; -W], Z = L11^-1 (unit lower triangular), W = L21 L11^-1, so the solves need
// no substitution inside a front: forward y = Z t1, v = t2 - W t1; backward x = Z^T D^-1 y - W^T x2.
#pragma once
#include <cuda_runtime.h>

#include <array>
#include <cstdint>
#include <memory>
#include <vector>

#include "dpf_direct.h"

namespace dpf {

constexpr long long kFrontMaxCells = 300000000;  // 32-bit cell and coupling numbers

struct Front {            // one tree node; positions 0..k-1 of its front are its own cells
    int first, k, m, pad; // own cells: first .. first + k - 1 in the new numbering
    int ch0, nch;         // children: child[ch0 .. ch0 + nch)
    long long rows;       // its u = m - k ancestor cells (ascending) and their positions in the
                          // parent's front: rows[] and rel[] from here
    long long panel;      // m x k column-major panel in the panel store
    long long upd;        // u x u column-major update matrix (lower part) in its level's pool
    long long vec;        // u entries of its update vector in the solves
    long long lbuf;       // large fronts: m x 16 block of L columns in the step buffer, then 16 x 16 Z, 16 pivots
};

// A dissection: cells in their new order and the tree in an order with children before parents.
struct Dissection {
    std::vector<int> perm;                    // new -> original
    std::vector<int> first, k, parent, depth; // per node
};
Dissection dissect_regular(const std::vector<std::array<int, 3>> &dims, const std::vector<long long> &off);
Dissection dissect_graph(int n, const std::vector<int> &rp, const std::vector<int> &ci);
// A band order cut into runs of kBandBlock rows, each the parent of the one before: its fronts have at most
// kBandBlock + w rows, whatever the graph.
constexpr int kBandBlock = 64;
Dissection dissect_band(const BandOrder &o);

// Fronts of a dissection for the couplings of a symmetric graph (CSR, original numbering).
struct FrontTree {
    std::vector<Front> fr;
    std::vector<int> child, rows, rel, node_of, depth;
    int max_depth = 0, max_m = 0;
    long long panel_size = 0, vec_size = 0, pool_size[2] = {0, 0}, lbuf_size = 0;
    double fma = 0;                           // multiply-adds of the factorisation
    double bytes() const;
};
// stops (returns false) once the fronts need more than max_bytes
bool build_fronts(const Dissection &d, const std::vector<int> &rp, const std::vector<int> &ci, double max_bytes,
                  FrontTree &t);
// the couplings of regular grids as such a graph
void regular_graph(const std::vector<std::array<int, 3>> &dims, const std::vector<long long> &off,
                   std::vector<int> &rp, std::vector<int> &ci);

// Where the entry of the (new) row r and column c, r >= c, of the operator goes.
struct FrontIndex {
    const Front *fr;
    const int *node_of, *rows;
    double *panels;
#ifdef __CUDACC__
    __device__ __forceinline__ double *at(int r, int c) const {
        const Front &f = fr[node_of[c]];
        int pos = r - f.first;
        if (pos >= f.k) {  // an ancestor's cell: its position among the ascending rows
            const int *R = rows + f.rows;
            int lo = 0, hi = f.m - f.k;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (R[mid] < r) lo = mid + 1;
                else hi = mid;
            }
            if (lo >= f.m - f.k || R[lo] != r) return nullptr;
            pos = f.k + lo;
        }
        return panels + f.panel + (long long)(c - f.first) * f.m + pos;
    }
#endif
};

// Raises the kernels' dynamic shared-memory limits, once per device, before any launch.
void configure_front_kernels();

class FrontSolver {
public:
    // a front's vector fits the shared memory of a block; above the cells of any graph within
    // direct_fits' limit whose separators are dense (w about n: n^3 <= 2e13)
    static constexpr int kMaxM = 28000;
    FrontSolver(const Dissection &d, const FrontTree &t, cudaStream_t stream);
    ~FrontSolver();
    FrontSolver(const FrontSolver &) = delete;
    FrontSolver &operator=(const FrontSolver &) = delete;

    const int *iperm() const { return d_iperm; }  // original row -> new row (device)
    FrontIndex index() const { return FrontIndex{d_fr, d_node_of, d_rows, d_panels}; }
    void clear();                             // zero the panels before a caller's kernel fills them
    bool factor();                            // false when a pivot is not positive
    void solve(const double *b, double *x);   // x = A^-1 b in the original numbering (device)
    // sqrt(sum (b - Ax)^2 / sum b^2) over the rows with dir[i] == 0 (a diagnostic of a solve; FP64
    // atomics, so the last bits may vary from run to run)
    double relres(const uint8_t *dir, const double *b, const double *Ax);
    void set_stream(cudaStream_t s) { stream = s; }
    long long launches = 0;

private:
    struct Level {
        int small0 = 0, nsmall = 0, large0 = 0, nlarge = 0;  // runs of the front lists
        int max_small_m = 0, max_large_m = 0, max_large_k = 0, max_large_nch = 0, max_child_u = 0;
        long long upd_large = 0;              // the large fronts' update matrices: pool[parity][0 .. upd_large)
    };
    cudaStream_t stream;
    int n = 0, max_depth = 0;
    std::vector<Level> lv;
    std::vector<void *> owned;
    Front *d_fr = nullptr;
    int *d_child = nullptr, *d_rows = nullptr, *d_rel = nullptr, *d_node_of = nullptr, *d_list = nullptr;
    int *d_perm = nullptr, *d_iperm = nullptr, *d_err = nullptr;
    double *d_panels = nullptr, *d_pool[2] = {nullptr, nullptr}, *d_vec = nullptr, *d_lbuf = nullptr;
    double *d_dinv = nullptr, *d_y = nullptr, *d_x = nullptr, *d_acc = nullptr;
    long long panel_size = 0;
};

// The fronts for a system that direct_fits accepted: those of its nested dissection within half the free
// memory, otherwise those of its band order within nine tenths of it. A dissection's fronts take less than the band
// but where the graph has no small separators: 8000 cells in two sets with couplings between the sets only want
// 18.8 GB, their band 0.5. False where neither fits.
bool choose_fronts(Dissection &d, const BandOrder &band, const std::vector<int> &rp, const std::vector<int> &ci,
                   size_t free_bytes, FrontTree &t);
std::unique_ptr<FrontSolver> make_fronts(Dissection d, const BandOrder &band, const std::vector<int> &rp,
                                         const std::vector<int> &ci, size_t free_bytes, cudaStream_t stream);

}  // namespace dpf
