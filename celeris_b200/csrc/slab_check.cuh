// The block elimination and norms of slab.cuh on their own, for tests of their edges: orders
// around the panel and lane counts, matrices without a pivot, NaN. Not part of any result path.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "runtime.cuh"
#include "slab.cuh"

namespace {

// W (n x ncol, ld) <- its elimination (gauss_jordan); ok, perm: its result. lost_warp >= 0: that
// warp's waits count as run out. intact: a failed elimination left what it does not own in
// shared memory as it was (perm2, and the flags of the columns behind the one without a pivot).
template <class T>
__global__ void __launch_bounds__(512) slab_check_solve(int n, int ncol, int ld, T* W, int inverse, int lost_warp,
                                                        int* perm, int* ok, int* intact) {
    extern __shared__ __align__(16) unsigned char smem[];
    cb::slab::Shared s = cb::slab::carve(smem, n);
    s.lost = lost_warp;
    constexpr int kMark = 0x5a5a5a5a;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s.perm2[i] = kMark;
    const bool got = cb::slab::gauss_jordan(n, ncol, W, ld, inverse != 0, s);
    __syncthreads();
    if (got)
        for (int i = threadIdx.x; i < n; i += blockDim.x) perm[i] = s.perm[i];
    ok[threadIdx.x] = got;
    if (threadIdx.x == 0) {
        int fine = 1;
        for (int i = 0; i < n; ++i) fine &= s.perm2[i] == kMark;
        bool behind = false;
        for (int j = 0; j < cb::slab::kNB; ++j) {
            if (behind) fine &= s.flag[j] == 0;
            behind = behind || (!got && s.flag[j] < 0);
        }
        *intact = fine;
    }
}

template <class T>
int run_solve(int n, int nrhs, int inverse, int threads, int lost_warp, const T* a, const T* b, T* x, T* ainv, int* ok_out) {
    const int c1 = sizeof(T) == sizeof(double) ? (n + 1) & ~1 : n;  // first right-hand side's column
    const int ncol = c1 + nrhs, ld = (ncol + 1) & ~1;
    std::vector<T> h((size_t)n * ld);
    std::memset(h.data(), 0, h.size() * sizeof(T));
    for (int i = 0; i < n; ++i) {
        std::copy(a + (size_t)i * n, a + (size_t)(i + 1) * n, h.begin() + (size_t)i * ld);
        std::copy(b + (size_t)i * nrhs, b + (size_t)(i + 1) * nrhs, h.begin() + (size_t)i * ld + c1);
    }
    const size_t bytes = h.size() * sizeof(T), words = (size_t)n + threads + 1;
    char* d = nullptr;
    CEL_TRY(celeris_rt::device_alloc(reinterpret_cast<void**>(&d), bytes + words * sizeof(int), "slab check"));
    T* dW = reinterpret_cast<T*>(d);
    int* dperm = reinterpret_cast<int*>(d + bytes);
    std::vector<int> hw(words);
    auto call = [&]() -> int {
        CEL_CUDA(cudaMemcpy(dW, h.data(), bytes, cudaMemcpyHostToDevice));
        CEL_CUDA(cudaMemset(dperm, 0, words * sizeof(int)));
        const size_t smem = cb::slab::shared_bytes(n);
        CEL_CUDA(cudaFuncSetAttribute(slab_check_solve<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        slab_check_solve<T><<<1, threads, smem>>>(n, ncol, ld, dW, inverse, lost_warp, dperm, dperm + n,
                                                   dperm + n + threads);
        celeris_rt::count_launch(1);
        CEL_CUDA(cudaGetLastError());
        CEL_CUDA(cudaMemcpy(h.data(), dW, bytes, cudaMemcpyDeviceToHost));
        CEL_CUDA(cudaMemcpy(hw.data(), dperm, words * sizeof(int), cudaMemcpyDeviceToHost));
        return CELERIS_OK;
    };
    const int status = call();
    cudaFree(d);
    CEL_TRY(status);
    const int* ok = hw.data() + n;
    *ok_out = ok[0];
    for (int t = 1; t < threads; ++t)
        if (ok[t] != ok[0]) return celeris_rt::set_error(CELERIS_ERR_CUDA, "threads disagree on the elimination's result");
    if (!ok[threads]) return celeris_rt::set_error(CELERIS_ERR_CUDA, "the elimination wrote outside its own arrays");
    if (!ok[0]) return CELERIS_OK;
    for (int k = 0; k < n; ++k) {
        const T* row = h.data() + (size_t)hw[k] * ld;
        std::copy(row + c1, row + c1 + nrhs, x + (size_t)k * nrhs);
        if (inverse)
            for (int l = 0; l < n; ++l) ainv[(size_t)k * n + hw[l]] = row[l];
    }
    return CELERIS_OK;
}

// out: norm_inf and max_entry of the n x n matrix A, as every thread has them (NaN if they differ).
__global__ void __launch_bounds__(512) slab_check_max(int n, const double* A, double* out) {
    __shared__ double red[32];
    __shared__ int differ;
    if (threadIdx.x == 0) differ = 0;
    const double a = cb::slab::norm_inf(n, A, n, red), b = cb::slab::max_entry(n, A, n, 0, red);
    __syncthreads();
    if (threadIdx.x == 0) {
        out[0] = a;
        out[1] = b;
    }
    __syncthreads();
    const auto same = [](double x, double y) { return x == y || (x != x && y != y); };
    if (!same(out[0], a) || !same(out[1], b)) atomicOr(&differ, 1);
    __syncthreads();
    if (threadIdx.x == 0) out[2] = differ;
}

}  // namespace

extern "C" int celeris_debug_slab_max(int n, int threads, const double* a, double* out) {
    CEL_TRY(celeris_rt::require_device());
    if (n < 1 || n > cb::slab::kMaxOrder || (threads != 256 && threads != 512) || !a || !out)
        return celeris_rt::set_error(CELERIS_ERR_INVALID_ARG, "n in [1, %d], threads 256 or 512", cb::slab::kMaxOrder);
    const size_t bytes = (size_t)n * n * sizeof(double);
    double* d = nullptr;
    double h[3];
    CEL_TRY(celeris_rt::device_alloc(reinterpret_cast<void**>(&d), bytes + sizeof(h), "slab check"));
    auto call = [&]() -> int {
        double* dout = d + (size_t)n * n;
        CEL_CUDA(cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice));
        slab_check_max<<<1, threads>>>(n, d, dout);
        celeris_rt::count_launch(1);
        CEL_CUDA(cudaGetLastError());
        CEL_CUDA(cudaMemcpy(h, dout, sizeof(h), cudaMemcpyDeviceToHost));
        return CELERIS_OK;
    };
    const int status = call();
    cudaFree(d);
    CEL_TRY(status);
    if (h[2] != 0.0) return celeris_rt::set_error(CELERIS_ERR_CUDA, "threads disagree on a block's maximum");
    out[0] = h[0];
    out[1] = h[1];
    return CELERIS_OK;
}

extern "C" int celeris_debug_slab_solve(int n, int nrhs, int is_complex, int inverse, int threads, int lost_warp,
                                        const double* a, const double* b, double* x, double* ainv, int* ok) {
    CEL_TRY(celeris_rt::require_device());
    // above order 256 the panel takes sixteen warps
    if (n < 1 || n > cb::slab::kMaxOrder || nrhs < 1 || (threads != 512 && (threads != 256 || n > 256)) || !a || !b ||
        !x || !ok || (inverse && !ainv))
        return celeris_rt::set_error(CELERIS_ERR_INVALID_ARG, "n in [1, %d], threads 256 (n <= 256) or 512",
                                     cb::slab::kMaxOrder);
    if (is_complex)
        return run_solve(n, nrhs, inverse, threads, lost_warp, reinterpret_cast<const cb::cplx*>(a),
                         reinterpret_cast<const cb::cplx*>(b), reinterpret_cast<cb::cplx*>(x), reinterpret_cast<cb::cplx*>(ainv), ok);
    return run_solve(n, nrhs, inverse, threads, lost_warp, a, b, x, ainv, ok);
}
