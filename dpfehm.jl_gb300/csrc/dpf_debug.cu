// dpf_debug.cu -- test hooks: the bounded waits of the staging kernels, the integer-only
// 48-bit split of doubles that the assembly and the round start use, the table-driven power and
// logarithm, and the band orderings of the direct solver (host code, callable without a GPU).
//
// dpf_debug_expired_wait runs one block whose threads wait on a shared-memory mbarrier
// that nothing arrives on, through the same bounded wait (mbar_wait) that every staging
// kernel uses, so that a test sees that wait end by its bound, the error word set and the
// device still usable, without any kernel of a solve being made to fail. dpf_debug_expired_barrier
// does the same for the grid barrier of the one-launch solves, with one block that never arrives.
#include <cuda_runtime.h>

#include <new>
#include <string>

#include "dpf_direct.h"
#include "dpf_front.h"
#include "dpf_grid.cuh"
#include "dpf_means.cuh"
#include "dpf_plane.cuh"

namespace dpf {

void set_global_error(const std::string &msg);

__global__ void k_expired_wait(int *err, unsigned long long *waited_ns) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);  // one arrival completes phase 0; none is made
    __syncthreads();
    const uint64_t t0 = global_ns();
    const bool done = mbar_wait(&bar, 0, err);
    __syncthreads();
    if (threadIdx.x == 0) {
        waited_ns[0] = global_ns() - t0;
        if (done) atomicExch(err, 2);  // the phase cannot complete: a defect of the wait
    }
}

// out: {error word, threads that saw the wait expire}, ns: the longest wait
__global__ void k_expired_barrier(unsigned *words, int *out, unsigned long long *ns, int with_last) {
    if (blockIdx.x == 0) return;  // never arrives
    GridBar bar{words, out};
    const uint64_t t0 = global_ns();
    const bool got = with_last ? bar.sync([] {}) : bar.sync();
    if (!got) atomicAdd(&out[1], 1);
    if (threadIdx.x == 0) atomicMax(ns, (unsigned long long)(global_ns() - t0));
}

__global__ void k_split48(long long n, const double *v, float *hi, float *lo, double *v48, int *ok) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float h = 0.f, l = 0.f;
    double w = 0.0;
    ok[i] = split48(v[i], h, l, w) ? 1 : 0;
    hi[i] = h;
    lo[i] = l;
    v48[i] = w;
}

__global__ void k_pow64(long long n, const double *x, const double *y, double *p, double *lhi, double *llo) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    LogDD l;
    p[i] = pow64(x[i], y[i], l);
    lhi[i] = l.hi;
    llo[i] = l.lo;
}

}  // namespace dpf

extern "C" int dpf_debug_pow64(int64_t n, const double *x, const double *y, double *p, double *log_hi, double *log_lo) {
    if (n < 0 || (n > 0 && (!x || !y || !p || !log_hi || !log_lo))) return DPF_BAD_INPUT;
    if (n == 0) return DPF_OK;
    dpf::k_pow64<<<(unsigned)((n + 255) / 256), 256>>>((long long)n, x, y, p, log_hi, log_lo);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaGetLastError();
        dpf::set_global_error(std::string("power probe: ") + cudaGetErrorString(e));
        return DPF_CUDA;
    }
    return DPF_OK;
}

extern "C" int dpf_debug_split48(int64_t n, const double *v, float *hi, float *lo, double *v48, int *ok) {
    if (n < 0 || (n > 0 && (!v || !hi || !lo || !v48 || !ok))) return DPF_BAD_INPUT;
    if (n == 0) return DPF_OK;
    dpf::k_split48<<<(unsigned)((n + 255) / 256), 256>>>((long long)n, v, hi, lo, v48, ok);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaGetLastError();
        dpf::set_global_error(std::string("split probe: ") + cudaGetErrorString(e));
        return DPF_CUDA;
    }
    return DPF_OK;
}

extern "C" int dpf_debug_expired_wait(double *waited_ms) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        dpf::set_global_error("no CUDA device");
        return DPF_NO_DEVICE;
    }
    void *buf = nullptr;
    if (dpf::dev_malloc(&buf, 16) != cudaSuccess) {
        cudaGetLastError();
        dpf::set_global_error("device allocation failed");
        return DPF_OOM;
    }
    int *d_err = (int *)buf;
    unsigned long long *d_ns = (unsigned long long *)((char *)buf + 8);
    int h_err = -1;
    unsigned long long h_ns = 0;
    cudaError_t e = cudaMemset(buf, 0, 16);
    if (e == cudaSuccess) {
        dpf::k_expired_wait<<<1, 32>>>(d_err, d_ns);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&h_ns, d_ns, sizeof(h_ns), cudaMemcpyDeviceToHost);
    dpf::dev_free(buf);
    if (e != cudaSuccess) {
        cudaGetLastError();
        dpf::set_global_error(std::string("expired-wait probe: ") + cudaGetErrorString(e));
        return DPF_CUDA;
    }
    if (waited_ms) *waited_ms = 1e-6 * (double)h_ns;
    if (h_err != 1) {
        dpf::set_global_error("the bounded wait did not report its expiry");
        return DPF_STATE;
    }
    dpf::set_global_error("a bounded staging wait expired after " + std::to_string(1e-6 * (double)h_ns) + " ms");
    return DPF_TIMEOUT;
}

extern "C" int dpf_debug_expired_barrier(int with_last, double *waited_ms) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        dpf::set_global_error("no CUDA device");
        return DPF_NO_DEVICE;
    }
    constexpr int kBlocks = 8, kThreads = 64;
    constexpr size_t kBytes = dpf::kGridBarWords * sizeof(unsigned) + 16;
    char *buf = nullptr;
    if (dpf::dev_malloc((void **)&buf, kBytes) != cudaSuccess) {
        cudaGetLastError();
        dpf::set_global_error("device allocation failed");
        return DPF_OOM;
    }
    unsigned *words = (unsigned *)buf;
    unsigned long long *d_ns = (unsigned long long *)(buf + dpf::kGridBarWords * sizeof(unsigned));
    int *d_out = (int *)(d_ns + 1);
    int h_out[2] = {-1, -1};
    unsigned long long h_ns = 0;
    void *args[] = {&words, &d_out, &d_ns, &with_last};
    cudaError_t e = cudaMemset(buf, 0, kBytes);
    if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel((const void *)dpf::k_expired_barrier, dim3(kBlocks), dim3(kThreads), args, 0, 0);
    if (e == cudaSuccess) e = cudaMemcpy(h_out, d_out, sizeof(h_out), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&h_ns, d_ns, sizeof(h_ns), cudaMemcpyDeviceToHost);
    dpf::dev_free(buf);
    if (e != cudaSuccess) {
        cudaGetLastError();
        dpf::set_global_error(std::string("expired-barrier probe: ") + cudaGetErrorString(e));
        return DPF_CUDA;
    }
    if (waited_ms) *waited_ms = 1e-6 * (double)h_ns;
    if (h_out[0] != 1 || h_out[1] != (kBlocks - 1) * kThreads) {
        dpf::set_global_error("the grid barrier did not report its expiry to every thread");
        return DPF_STATE;
    }
    dpf::set_global_error("a grid barrier expired after " + std::to_string(1e-6 * (double)h_ns) + " ms");
    return DPF_TIMEOUT;
}

// The direct solver's band orderings, run on the host: perm[k] = the original row of band row k,
// *w = the half-bandwidth the ordering gives.
extern "C" int dpf_debug_band_order_graph(int64_t n, const int32_t *rp, const int32_t *ci, int64_t *perm,
                                          int64_t *w) {
    if (n < 0 || !rp || !perm || !w || n > (int64_t)1 << 30) return DPF_BAD_INPUT;
    if (rp[0] != 0) return DPF_BAD_INPUT;
    for (int64_t i = 0; i < n; i++)
        if (rp[i + 1] < rp[i]) return DPF_BAD_INPUT;
    const int64_t nnz = rp[n];
    if (nnz > 0 && !ci) return DPF_BAD_INPUT;
    for (int64_t e = 0; e < nnz; e++)
        if (ci[e] < 0 || ci[e] >= n) return DPF_BAD_INPUT;
    try {
        std::vector<int> r(rp, rp + n + 1), c(ci, ci + nnz);
        const dpf::BandOrder o = dpf::band_order_rcm((long long)n, r, c);
        for (int64_t k = 0; k < n; k++) perm[k] = o.perm[k];
        *w = o.w;
    } catch (const std::bad_alloc &) {
        return DPF_OOM;
    }
    return DPF_OK;
}

extern "C" int dpf_debug_direct_fronts(int64_t n, const int32_t *rp, const int32_t *ci, int64_t free_bytes, int *form,
                                       int64_t *max_rows, double *bytes) {
    if (n < 1 || n >= dpf::kFrontMaxCells || !rp || !form || !max_rows || !bytes || free_bytes < 0) return DPF_BAD_INPUT;
    if (rp[0] != 0) return DPF_BAD_INPUT;
    for (int64_t i = 0; i < n; i++)
        if (rp[i + 1] < rp[i]) return DPF_BAD_INPUT;
    if (rp[n] > 0 && !ci) return DPF_BAD_INPUT;
    for (int32_t e = 0; e < rp[n]; e++)
        if (ci[e] < 0 || ci[e] >= n) return DPF_BAD_INPUT;
    try {
        std::vector<int> r(rp, rp + n + 1), c(ci, ci + rp[n]);
        const dpf::BandOrder band = dpf::band_order_rcm((long long)n, r, c);
        *form = 0;
        *max_rows = 0;
        *bytes = 0.0;
        if (!dpf::direct_fits((long long)n, band.w, (size_t)free_bytes / 2)) return DPF_OK;
        dpf::Dissection d = dpf::dissect_graph((int)n, r, c);
        const size_t nodes = d.k.size();
        const std::vector<int> perm = d.perm;
        dpf::FrontTree t;
        const bool fits = dpf::choose_fronts(d, band, r, c, (size_t)free_bytes, t);
        *form = !fits ? -1 : d.k.size() == nodes && d.perm == perm ? 1 : 2;
        *max_rows = t.max_m;
        *bytes = t.bytes();
    } catch (const std::bad_alloc &) {
        return DPF_OOM;
    }
    return DPF_OK;
}

extern "C" int dpf_debug_band_order_grids(int nprob, const int32_t *dims, int64_t *perm, int64_t *w) {
    if (nprob < 0 || (nprob > 0 && !dims) || !perm || !w) return DPF_BAD_INPUT;
    try {
        std::vector<std::array<int, 3>> d(nprob);
        std::vector<long long> off(nprob);
        long long n = 0;
        for (int p = 0; p < nprob; p++) {
            for (int a = 0; a < 3; a++) {
                if (dims[3 * p + a] < 1) return DPF_BAD_INPUT;
                d[p][a] = dims[3 * p + a];
            }
            off[p] = n;
            n += (long long)d[p][0] * d[p][1] * d[p][2];
            if (n > (1LL << 30)) return DPF_BAD_INPUT;
        }
        const dpf::BandOrder o = dpf::band_order_regular(d, off);
        for (long long k = 0; k < n; k++) perm[k] = o.perm[k];
        *w = o.w;
    } catch (const std::bad_alloc &) {
        return DPF_OOM;
    }
    return DPF_OK;
}
