// dpf_direct.h -- which systems the direct solver behind `linear_solver = cholesky_solver`
// (src/groundwater.jl:56-60, which calls LinearAlgebra.cholesky on the assembled sparse matrix) takes.
//
// The measure is the half-bandwidth w of a band ordering of the rows (regular grids: the two shortest
// axes fastest; other meshes: reverse Cuthill-McKee): 2-D grids, thin 3-D grids and moderate meshes have
// n (w + 1) values and n w^2 multiply-adds within reach, and are factored by dpf_front.h; wider
// ones are refused and the caller takes its iterative solve to the rounding floor instead.
#pragma once
#include <array>
#include <cstdint>
#include <vector>

namespace dpf {

// A band ordering: perm[k] = original row of band row k, and the half-bandwidth w = the largest
// |k_i - k_j| over the couplings (i, j).
struct BandOrder {
    std::vector<long long> perm;
    long long w = 0;
};

// The cells of a batch of regular grids (problem p: dims[p] = {nx, ny, nz}, z fastest, its
// cells from off[p]): per problem the axes re-nested by extent (the longest slowest), problems
// one after another; w = the largest product of a problem's two shorter extents.
BandOrder band_order_regular(const std::vector<std::array<int, 3>> &dims, const std::vector<long long> &off);

// A symmetric graph in CSR form (rp[n + 1], ci; no diagonal): reverse Cuthill-McKee, each
// connected component started from a pseudo-peripheral vertex (the last one reached by a
// breadth-first search from its lowest-degree vertex).
BandOrder band_order_rcm(long long n, const std::vector<int> &rp, const std::vector<int> &ci);

// whether the direct solver takes a system: a band of n (w + 1) doubles within `mem_bytes`, and at most
// 2e13 for n w^2
bool direct_fits(long long n, long long w, size_t mem_bytes);

}  // namespace dpf
