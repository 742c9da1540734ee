// What a batch needs before its search, on the GPU in one launch each: the checks and statistics of
// device-resident queries (the reference's _validation.as_matrix and metrics.prepare checks, and the
// inputs of the choice of distance arithmetic), the bitmap of a filter mask, and code-space queries
// (quantization.py:61-68). As separate tensor operations the query checks alone were 25 launches with a
// read-back, about 330 us before a 10K batch's 3 ms search.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <string>

#include "hnsw_b200.h"

namespace hb {
int fail(int code, const std::string &msg);
}

namespace hbq {

constexpr int THREADS = 256;
constexpr int PER_THREAD = 16;  // elements a thread reads before its block reduces
constexpr int MAX_BLOCKS = 592;

// Order-preserving key of a double (never 0 for a number), and back.
__host__ __device__ inline unsigned long long key_of(double d) {
    union {
        double d;
        unsigned long long u;
    } c;
    c.d = d;
    return (c.u >> 63) ? ~c.u : (c.u | 0x8000000000000000ull);
}
inline double value_of(unsigned long long k) {
    union {
        double d;
        unsigned long long u;
    } c;
    c.u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return c.d;
}

// work[0]: flags; work[1]: largest key; work[2]: largest complemented key (the smallest); all zeroed.
template <typename T>
__global__ void __launch_bounds__(THREADS) stats_kernel(const T *__restrict__ raw, const float *__restrict__ rows,
                                                        int64_t count, const double *__restrict__ norms,
                                                        int64_t n_norms, unsigned long long *work) {
    unsigned f = 0;
    double lo = INFINITY, hi = -INFINITY;
    const int64_t at = int64_t(blockIdx.x) * THREADS + threadIdx.x, step = int64_t(gridDim.x) * THREADS;
    auto see = [&](double v) {
        if (!(fabs(v) <= DBL_MAX)) f |= HNSW_B200_ROWS_NOT_FINITE;
        if (v != rint(v)) f |= HNSW_B200_NOT_INTEGER;
        lo = fmin(lo, v);
        hi = fmax(hi, v);
    };
#pragma unroll 4
    for (int64_t i = at; i < count; i += step) {
        const double v = double(raw[i]);
        if (!(fabs(v) <= DBL_MAX)) f |= HNSW_B200_NOT_FINITE;
        see(rows ? double(rows[i]) : v);
    }
    for (int64_t i = at; i < n_norms; i += step)
        if (norms[i] == 0.0) f |= HNSW_B200_ZERO_NORM;
    unsigned long long a = key_of(hi), b = ~key_of(lo);
    f = __reduce_or_sync(0xffffffffu, f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    __shared__ unsigned sf[THREADS / 32];
    __shared__ unsigned long long sa[THREADS / 32], sb[THREADS / 32];
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        sf[warp] = f;
        sa[warp] = a;
        sb[warp] = b;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < THREADS / 32; w++) {
        f |= sf[w];
        a = max(a, sa[w]);
        b = max(b, sb[w]);
    }
    if (f) atomicOr(reinterpret_cast<unsigned *>(work), f);
    atomicMax(work + 1, a);
    atomicMax(work + 2, b);
}

// Bit i of the bitmap: mask[node_ids[i]] (mask[i] without an order); one word a warp.
__global__ void __launch_bounds__(THREADS) pack_mask_kernel(const uint8_t *__restrict__ mask,
                                                            const int32_t *__restrict__ node_ids, int64_t n,
                                                            uint32_t *__restrict__ bits) {
    const int64_t i = int64_t(blockIdx.x) * THREADS + threadIdx.x;
    const bool in = i < n;
    const uint32_t w = __ballot_sync(0xffffffffu, in && mask[in && node_ids ? node_ids[i] : (in ? i : 0)] != 0);
    if ((threadIdx.x & 31) == 0 && in) bits[i >> 5] = w;
}

__global__ void __launch_bounds__(THREADS) code_queries_kernel(const float *__restrict__ x, int64_t count, int32_t dim,
                                                               const double *__restrict__ offset, double step,
                                                               double *__restrict__ out) {
    for (int64_t i = int64_t(blockIdx.x) * THREADS + threadIdx.x; i < count; i += int64_t(gridDim.x) * THREADS) {
        const double v = double(x[i]);
        out[i] = offset ? __ddiv_rn(__dsub_rn(v, offset[i % dim]), step) : v;
    }
}

int blocks_for(int64_t count, int per_thread) {
    return int(std::max<int64_t>(1, std::min<int64_t>(MAX_BLOCKS, (count + THREADS * per_thread - 1) /
                                                                       (int64_t(THREADS) * per_thread))));
}

int done(const char *what) {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? HNSW_B200_OK
                            : hb::fail(HNSW_B200_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace hbq

extern "C" int hnsw_b200_device_stats(const void *raw, int32_t float64, const float *rows, int64_t count,
                                      const double *norms, int64_t n_norms, void *work, uint32_t *flags,
                                      hnsw_b200_value_stats_t *out, void *stream) {
    using namespace hbq;
    if (count < 0 || n_norms < 0 || !work || !flags || !out || (count > 0 && !raw) || (n_norms > 0 && !norms))
        return hb::fail(HNSW_B200_EINVAL, "device_stats: bad argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto *w = static_cast<unsigned long long *>(work);
    cudaMemsetAsync(w, 0, 24, s);
    const int blocks = blocks_for(count, PER_THREAD);
    if (float64)
        stats_kernel<double><<<blocks, THREADS, 0, s>>>(static_cast<const double *>(raw), rows, count, norms, n_norms, w);
    else
        stats_kernel<float><<<blocks, THREADS, 0, s>>>(static_cast<const float *>(raw), rows, count, norms, n_norms, w);
    unsigned long long h[3] = {0, 0, 0};
    cudaMemcpyAsync(h, w, 24, cudaMemcpyDeviceToHost, s);
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return hb::fail(HNSW_B200_ECUDA, std::string("device_stats: ") + cudaGetErrorString(e));
    if (int rc = done("device_stats")) return rc;
    *flags = uint32_t(h[0]);
    out->finite = (*flags & (HNSW_B200_NOT_FINITE | HNSW_B200_ROWS_NOT_FINITE)) == 0;
    out->integer = (*flags & HNSW_B200_NOT_INTEGER) == 0;
    out->max = count ? value_of(h[1]) : 0.0;
    out->min = count ? value_of(~h[2]) : 0.0;
    return HNSW_B200_OK;
}

extern "C" int hnsw_b200_pack_mask(const uint8_t *mask, const int32_t *node_ids, int64_t n, uint32_t *bits,
                                   void *stream) {
    using namespace hbq;
    if (n < 0 || (n > 0 && (!mask || !bits))) return hb::fail(HNSW_B200_EINVAL, "pack_mask: bad argument");
    if (n == 0) return HNSW_B200_OK;
    pack_mask_kernel<<<unsigned((n + THREADS - 1) / THREADS), THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
        mask, node_ids, n, bits);
    return done("pack_mask");
}

extern "C" int hnsw_b200_code_queries(const float *queries, int64_t nq, int32_t dim, const double *offset, double step,
                                      double *out, void *stream) {
    using namespace hbq;
    if (nq < 0 || dim < 1 || (nq > 0 && (!queries || !out)))
        return hb::fail(HNSW_B200_EINVAL, "code_queries: bad argument");
    if (nq == 0) return HNSW_B200_OK;
    code_queries_kernel<<<blocks_for(nq * dim, 4), THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
        queries, nq * dim, dim, offset, step, out);
    return done("code_queries");
}
