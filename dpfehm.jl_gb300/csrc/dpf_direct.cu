// dpf_direct.cu -- band orderings and the size limit of the direct solver (see dpf_direct.h).
#include "dpf_direct.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace dpf {

BandOrder band_order_regular(const std::vector<std::array<int, 3>> &dims, const std::vector<long long> &off) {
    BandOrder o;
    long long n = 0;
    for (size_t p = 0; p < dims.size(); p++) n = std::max(n, off[p] + (long long)dims[p][0] * dims[p][1] * dims[p][2]);
    o.perm.assign(n, 0);
    for (size_t p = 0; p < dims.size(); p++) {
        const int nn[3] = {dims[p][0], dims[p][1], dims[p][2]};
        const long long st[3] = {(long long)nn[1] * nn[2], nn[2], 1};
        int ax[3] = {0, 1, 2};
        std::stable_sort(ax, ax + 3, [&](int a, int b) { return nn[a] > nn[b]; });  // longest slowest
        const long long w = (long long)nn[ax[1]] * nn[ax[2]];
        if (nn[ax[0]] > 1) o.w = std::max(o.w, w);
        else if (nn[ax[1]] > 1) o.w = std::max(o.w, (long long)nn[ax[2]]);
        else if (nn[ax[2]] > 1) o.w = std::max(o.w, 1LL);
        long long k = off[p];
        for (int a = 0; a < nn[ax[0]]; a++)
            for (int b = 0; b < nn[ax[1]]; b++)
                for (int c = 0; c < nn[ax[2]]; c++)
                    o.perm[k++] = off[p] + a * st[ax[0]] + b * st[ax[1]] + c * st[ax[2]];
    }
    return o;
}

BandOrder band_order_rcm(long long n, const std::vector<int> &rp, const std::vector<int> &ci) {
    BandOrder o;
    std::vector<int> deg(n);
    for (long long i = 0; i < n; i++) deg[i] = rp[i + 1] - rp[i];
    std::vector<char> seen(n, 0);
    std::vector<long long> order;
    order.reserve(n);
    std::vector<int> level(n, -1);
    // breadth-first levels from s over the unvisited component; returns the vertex of smallest
    // degree in the deepest level
    auto bfs_far = [&](long long s, std::vector<long long> &comp) {
        comp.clear();
        comp.push_back(s);
        level[s] = 0;
        for (size_t h = 0; h < comp.size(); h++) {
            const long long v = comp[h];
            for (int e = rp[v]; e < rp[v + 1]; e++) {
                const int u = ci[e];
                if (u != v && level[u] < 0 && !seen[u]) {
                    level[u] = level[v] + 1;
                    comp.push_back(u);
                }
            }
        }
        long long best = comp.back();
        for (long long v : comp)
            if (level[v] == level[comp.back()] && deg[v] < deg[best]) best = v;
        for (long long v : comp) level[v] = -1;
        return best;
    };
    std::vector<long long> comp;
    std::vector<int> nb;
    for (long long s0 = 0; s0 < n; s0++) {
        if (seen[s0]) continue;
        // pseudo-peripheral start: twice the farthest lowest-degree vertex
        long long s = bfs_far(s0, comp);
        s = bfs_far(s, comp);
        // Cuthill-McKee from s: neighbours in order of increasing degree
        const size_t first = order.size();
        order.push_back(s);
        seen[s] = 1;
        for (size_t h = first; h < order.size(); h++) {
            const long long v = order[h];
            nb.clear();
            for (int e = rp[v]; e < rp[v + 1]; e++)
                if (!seen[ci[e]] && ci[e] != v) {
                    seen[ci[e]] = 1;
                    nb.push_back(ci[e]);
                }
            std::sort(nb.begin(), nb.end(), [&](int a, int b) { return deg[a] < deg[b] || (deg[a] == deg[b] && a < b); });
            for (int u : nb) order.push_back(u);
        }
        std::reverse(order.begin() + first, order.end());
    }
    o.perm = order;
    std::vector<long long> pos(n);
    for (long long k = 0; k < n; k++) pos[order[k]] = k;
    for (long long i = 0; i < n; i++)
        for (int e = rp[i]; e < rp[i + 1]; e++) o.w = std::max(o.w, std::llabs(pos[i] - pos[ci[e]]));
    return o;
}

bool direct_fits(long long n, long long w, size_t mem_bytes) {
    if (n <= 0) return false;
    const double bytes = 8.0 * (double)n * (double)(w + 1) + 24.0 * (double)n;
    return bytes <= (double)mem_bytes && (double)n * (double)w * (double)w <= 2e13;
}

}  // namespace dpf
