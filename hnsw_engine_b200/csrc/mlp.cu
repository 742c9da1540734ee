// Training and packing of the early-termination network: 12 -> 64 -> 64 -> 1, ReLU.
//
// The network has no reference counterpart (it is the learned part of this engine). Training keeps
// float32 master weights and runs the forward pass with BF16-rounded weights and FP32
// accumulation -- exactly the arithmetic of the in-search inference (search.cu, mlp_eval) -- so the
// trained network behaves identically when it is packed and used by the search kernel.
//
// Master parameter vector (float32, MLP_PARAMS values):
//   W1 [64][12] | b1 [64] | W2 [64][64] | b2 [64] | W3 [64] | b3 [1]
// Loss: mean squared error of the prediction against log1p(remaining checkpoints).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include "hnsw_b200.h"

namespace hb {
int fail(int code, const std::string &msg);
}

namespace hbm {

constexpr int F = HNSW_B200_STOP_FEATURES;  // 12
constexpr int H = HNSW_B200_STOP_HIDDEN;    // 64
constexpr int O_W1 = 0;
constexpr int O_B1 = O_W1 + H * F;
constexpr int O_W2 = O_B1 + H;
constexpr int O_B2 = O_W2 + H * H;
constexpr int O_W3 = O_B2 + H;
constexpr int O_B3 = O_W3 + H;
constexpr int NPARAM = O_B3 + 1;  // 5057
constexpr unsigned FULL = 0xffffffffu;
// Shared-memory copy with padded row strides (13 and 65 words) so that lane j reading row j is
// bank-conflict free.
constexpr int S_W1 = 13, S_W2 = 65;
constexpr int SMEM_FLOATS = H * S_W1 + H + H * S_W2 + H + H + 1;

__device__ __forceinline__ float bf(float w) { return __bfloat162float(__float2bfloat16_rn(w)); }

__device__ void load_weights(const float *P, float *s) {
    float *w1 = s, *b1 = w1 + H * S_W1, *w2 = b1 + H, *b2 = w2 + H * S_W2, *w3 = b2 + H, *b3 = w3 + H;
    for (int i = threadIdx.x; i < H * F; i += blockDim.x) w1[(i / F) * S_W1 + i % F] = bf(P[O_W1 + i]);
    for (int i = threadIdx.x; i < H * H; i += blockDim.x) w2[(i / H) * S_W2 + i % H] = bf(P[O_W2 + i]);
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        b1[i] = P[O_B1 + i];
        b2[i] = P[O_B2 + i];
        w3[i] = bf(P[O_W3 + i]);
    }
    if (threadIdx.x == 0) b3[0] = P[O_B3];
    __syncthreads();
}

// Forward of one sample by one warp: h1 (lanes j, j+32), h2 (lanes j, j+32), output (all lanes).
__device__ __forceinline__ float forward(const float *s, const float *x, int lane, float &h1a,
                                         float &h1b, float &h2a, float &h2b) {
    const float *w1 = s, *b1 = w1 + H * S_W1, *w2 = b1 + H, *b2 = w2 + H * S_W2, *w3 = b2 + H, *b3 = w3 + H;
    h1a = b1[lane];
    h1b = b1[lane + 32];
#pragma unroll
    for (int i = 0; i < F; i++) {
        h1a = fmaf(w1[lane * S_W1 + i], x[i], h1a);
        h1b = fmaf(w1[(lane + 32) * S_W1 + i], x[i], h1b);
    }
    h1a = fmaxf(h1a, 0.f);
    h1b = fmaxf(h1b, 0.f);
    h2a = b2[lane];
    h2b = b2[lane + 32];
#pragma unroll 8
    for (int i = 0; i < 32; i++) {
        const float u = __shfl_sync(FULL, h1a, i), v = __shfl_sync(FULL, h1b, i);
        h2a = fmaf(w2[lane * S_W2 + i], u, h2a);
        h2b = fmaf(w2[(lane + 32) * S_W2 + i], u, h2b);
        h2a = fmaf(w2[lane * S_W2 + 32 + i], v, h2a);
        h2b = fmaf(w2[(lane + 32) * S_W2 + 32 + i], v, h2b);
    }
    h2a = fmaxf(h2a, 0.f);
    h2b = fmaxf(h2b, 0.f);
    float o = w3[lane] * h2a + w3[lane + 32] * h2b;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) o += __shfl_xor_sync(FULL, o, off);
    return o + b3[0];
}

// Per-sample forward and backward: activations and their gradients for the reduction kernel.
__global__ void mlp_fwd_bwd(const float *P, const float *X, const float *Y, int B, float *H1,
                            float *H2, float *dH1, float *dH2, float *dO, float *loss) {
    extern __shared__ float sw[];
    load_weights(P, sw);
    const float *w2 = sw + H * S_W1 + H, *w3 = w2 + H * S_W2 + H;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    float lsum = 0.f;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < B; b += warps) {
        float x[F];
#pragma unroll
        for (int i = 0; i < F; i++) x[i] = X[int64_t(b) * F + i];
        float h1a, h1b, h2a, h2b;
        const float o = forward(sw, x, lane, h1a, h1b, h2a, h2b);
        const float err = o - Y[b];
        const float g = 2.f * err / float(B);
        lsum += err * err / float(B);
        const float g2a = h2a > 0.f ? g * w3[lane] : 0.f;
        const float g2b = h2b > 0.f ? g * w3[lane + 32] : 0.f;
        // dh1[i] = sum_j W2[j][i] dh2[j]; lane i holds i and i + 32.
        float g1a = 0.f, g1b = 0.f;
#pragma unroll 8
        for (int j = 0; j < 32; j++) {
            const float u = __shfl_sync(FULL, g2a, j), v = __shfl_sync(FULL, g2b, j);
            g1a = fmaf(w2[j * S_W2 + lane], u, g1a);
            g1b = fmaf(w2[j * S_W2 + lane + 32], u, g1b);
            g1a = fmaf(w2[(j + 32) * S_W2 + lane], v, g1a);
            g1b = fmaf(w2[(j + 32) * S_W2 + lane + 32], v, g1b);
        }
        g1a = h1a > 0.f ? g1a : 0.f;
        g1b = h1b > 0.f ? g1b : 0.f;
        const int64_t r = int64_t(b) * H;
        H1[r + lane] = h1a;
        H1[r + lane + 32] = h1b;
        H2[r + lane] = h2a;
        H2[r + lane + 32] = h2b;
        dH1[r + lane] = g1a;
        dH1[r + lane + 32] = g1b;
        dH2[r + lane] = g2a;
        dH2[r + lane + 32] = g2b;
        if (lane == 0) dO[b] = g;
    }
    if (lane == 0 && lsum != 0.f) atomicAdd(loss, lsum);
}

// Weight gradients dW1 = dH1^T X, dW2 = dH2^T H1, dW3 = dO^T H2, biases the column sums: every parameter
// is summed over the batch by one thread, sample after sample (deterministic, and the order in which the
// shipped networks were trained). What bounds that is the chain of one fused multiply-add a sample,
// four cycles each, so the samples must be at hand: a block owns parameters that share columns, copies
// those columns of 64 samples at a time into shared memory with cp.async, GRAD_STAGES - 1 chunks ahead, by
// four warps of its own (one warp a scheduler adds, and would not hide the copies' instructions either). With each thread loading from memory as it went, a batch of 4,096
// took 182 us; this takes 35, the Adam step included.
//  blocks 0..15: W2 rows 4 r .. 4 r + 3, two a thread (H1 whole, four columns of dH2);
//  16..21: W1 columns 2 r, 2 r + 1 (dH1 whole, X);  22: b1;  23: b2;  24: W3 and b3 (H2 whole, dO).
// G != NULL: the gradients are written there. Else one Adam step (Kingma & Ba) with bias correction on the
// float32 masters.
constexpr int GRAD_CHUNK = 64, GRAD_STAGES = 4, ADD_THREADS = 128, GRAD_THREADS = 256, GRAD_BLOCKS = 25;
constexpr int COPY_THREADS = GRAD_THREADS - ADD_THREADS;
constexpr int GRAD_S2 = 16;  // floats a sample of the second array: 4 (dH2), 12 (X) or 1 (dO)
constexpr int GRAD_STAGE_FLOATS = GRAD_CHUNK * (H + GRAD_S2);

struct AdamArgs {
    float *P, *M, *V;
    float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ void copy_async(float *dst, const float *src, bool by16) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if (by16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// count contiguous floats, by the copying threads
__device__ __forceinline__ void copy_run(float *dst, const float *src, int count, bool by16) {
    const int t = threadIdx.x - ADD_THREADS, n4 = by16 ? count >> 2 : 0;
    for (int e = t; e < n4; e += COPY_THREADS) copy_async(dst + 4 * e, src + 4 * e, true);
    for (int e = 4 * n4 + t; e < count; e += COPY_THREADS) copy_async(dst + e, src + e, false);
}

// add(load(b)) for the nb samples of a chunk, in order. A whole chunk goes 16 samples at a time, the next
// 16 read from shared memory while the multiply-adds of the current ones run (one warp a scheduler: nothing
// else hides the reads).
template <class Load, class Add>
__device__ __forceinline__ void each_sample(int nb, Load load, Add add) {
    if (nb == GRAD_CHUNK) {
        constexpr int R = 16;
        decltype(load(0)) v[2][R];
#pragma unroll
        for (int i = 0; i < R; i++) v[0][i] = load(i);
#pragma unroll
        for (int k = 0; k < GRAD_CHUNK / R; k++) {
            if (k + 1 < GRAD_CHUNK / R) {
#pragma unroll
                for (int i = 0; i < R; i++) v[(k + 1) & 1][i] = load((k + 1) * R + i);
            }
#pragma unroll
            for (int i = 0; i < R; i++) add(v[k & 1][i]);
        }
    } else {
        for (int b = 0; b < nb; b++) add(load(b));
    }
}

__global__ void __launch_bounds__(GRAD_THREADS) mlp_grads(const float *X, const float *H1, const float *H2,
                                                          const float *dH1, const float *dH2, const float *dO,
                                                          int B, float *G, const AdamArgs A) {
    extern __shared__ __align__(16) float st[];
    const int t = threadIdx.x, blk = blockIdx.x;
    const bool is_w2 = blk < 16, is_w1 = blk >= 16 && blk < 22, is_w3 = blk == 24;
    const float *s1 = is_w2 ? H1 : is_w3 ? H2 : blk == 23 ? dH2 : dH1;
    const float *s2 = is_w2 ? dH2 + 4 * blk : is_w1 ? X : dO;
    const int w2 = is_w1 ? F : is_w3 ? 1 : 0;  // floats a sample, contiguous (W2: four of H)
    const bool by16 = ((reinterpret_cast<uintptr_t>(s1) | reinterpret_cast<uintptr_t>(s2)) & 15) == 0;
    const int chunks = (B + GRAD_CHUNK - 1) / GRAD_CHUNK;
    auto fetch = [&](int c) {
        if (c < chunks) {
            float *d1 = st + (c % GRAD_STAGES) * GRAD_STAGE_FLOATS, *d2 = d1 + GRAD_CHUNK * H;
            const int b0 = c * GRAD_CHUNK, nb = min(GRAD_CHUNK, B - b0);
            copy_run(d1, s1 + int64_t(b0) * H, nb * H, by16);
            if (is_w2) {  // four of the columns
                for (int e = t - ADD_THREADS; e < (by16 ? nb : 4 * nb); e += COPY_THREADS) {
                    const int r = by16 ? e : e >> 2, o = by16 ? 0 : e & 3;
                    copy_async(d2 + 4 * r + o, s2 + int64_t(b0 + r) * H + o, by16);
                }
            } else if (w2) {
                copy_run(d2, s2 + int64_t(b0) * w2, nb * w2, by16);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const bool copies = t >= ADD_THREADS;
    for (int c = 0; c < GRAD_STAGES - 1 && copies; c++) fetch(c);
    const int col = t & 63, half = t >> 6;
    float acc0 = 0.f, acc1 = 0.f;
    for (int c = 0; c < chunks; c++) {
        if (copies) asm volatile("cp.async.wait_group %0;" ::"n"(GRAD_STAGES - 2) : "memory");
        __syncthreads();  // chunk c is there, and every thread is done with the chunk fetched over next
        if (copies) {
            fetch(c + GRAD_STAGES - 1);
            continue;
        }
        const float *d1 = st + (c % GRAD_STAGES) * GRAD_STAGE_FLOATS, *d2 = d1 + GRAD_CHUNK * H;
        const int nb = min(GRAD_CHUNK, B - c * GRAD_CHUNK);
        if (is_w2) {
            each_sample(nb, [&](int b) {
                const float2 d = *reinterpret_cast<const float2 *>(d2 + b * 4 + 2 * half);
                return make_float3(d1[b * H + col], d.x, d.y);
            }, [&](float3 v) {
                acc0 = fmaf(v.y, v.x, acc0);
                acc1 = fmaf(v.z, v.x, acc1);
            });
        } else if (is_w1) {
            const int i = 2 * (blk - 16) + half;
            each_sample(nb, [&](int b) { return make_float2(d1[b * H + col], d2[b * F + i]); },
                        [&](float2 v) { acc0 = fmaf(v.x, v.y, acc0); });
        } else if (is_w3 && half == 0) {
            each_sample(nb, [&](int b) { return make_float2(d2[b], d1[b * H + col]); },
                        [&](float2 v) { acc0 = fmaf(v.x, v.y, acc0); });
        } else if (is_w3 ? col == 0 : half == 0) {
            each_sample(nb, [&](int b) { return is_w3 ? d2[b] : d1[b * H + col]; }, [&](float v) { acc0 += v; });
        }
    }
    if (copies) return;
    auto finish = [&](int p, float g) {
        if (G) {
            G[p] = g;
            return;
        }
        const float m = A.b1 * A.M[p] + (1.f - A.b1) * g;
        const float v = A.b2 * A.V[p] + (1.f - A.b2) * g * g;
        A.M[p] = m;
        A.V[p] = v;
        A.P[p] -= A.lr * (m / A.c1) / (sqrtf(v / A.c2) + A.eps);
    };
    if (is_w2) {
        const int j = 4 * blk + 2 * half;
        finish(O_W2 + j * H + col, acc0);
        finish(O_W2 + (j + 1) * H + col, acc1);
    } else if (is_w1) {
        finish(O_W1 + col * F + 2 * (blk - 16) + half, acc0);
    } else if (is_w3) {
        if (half == 0) finish(O_W3 + col, acc0);
        else if (col == 0) finish(O_B3, acc0);
    } else if (half == 0) {
        finish((blk == 22 ? O_B1 : O_B2) + col, acc0);
    }
}

__global__ void mlp_predict_kernel(const float *P, const float *X, int n, float *out) {
    extern __shared__ float sw[];
    load_weights(P, sw);
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < n; b += warps) {
        float x[F];
#pragma unroll
        for (int i = 0; i < F; i++) x[i] = X[int64_t(b) * F + i];
        float h1a, h1b, h2a, h2b;
        const float o = forward(sw, x, lane, h1a, h1b, h2a, h2b);
        if (lane == 0) out[b] = o;
    }
}

// Inference layout used by the search kernel: bf16 W1, W2 and W3 in lane pairs, then float32 b1 [64],
// b2 [64], b3 [1], feature mean [12], feature 1/std [12]. A pair is the weights of hidden units l and
// l + 32 for one input, (W[l][i], W[l + 32][i]), stored at [i][l]: lane l reads both of its units'
// weights for input i in one 32-bit load.
__global__ void mlp_pack_kernel(const float *P, const float *mean, const float *inv_std,
                                unsigned char *dst) {
    __nv_bfloat16 *w = reinterpret_cast<__nv_bfloat16 *>(dst);
    float *b = reinterpret_cast<float *>(dst + size_t(H * F + H * H + H) * 2);
    for (int t = threadIdx.x; t < H * F; t += blockDim.x) {
        const int i = t / H, j = (t % H) / 2 + 32 * (t % 2);  // pair [i][l], half -> unit j
        w[t] = __float2bfloat16_rn(P[O_W1 + j * F + i]);
    }
    for (int t = threadIdx.x; t < H * H; t += blockDim.x) {
        const int i = t / H, j = (t % H) / 2 + 32 * (t % 2);
        w[H * F + t] = __float2bfloat16_rn(P[O_W2 + j * H + i]);
    }
    for (int t = threadIdx.x; t < H; t += blockDim.x) {
        w[H * F + H * H + t] = __float2bfloat16_rn(P[O_W3 + t / 2 + 32 * (t % 2)]);
        b[t] = P[O_B1 + t];
        b[H + t] = P[O_B2 + t];
    }
    if (threadIdx.x == 0) b[2 * H] = P[O_B3];
    for (int t = threadIdx.x; t < F; t += blockDim.x) {
        b[2 * H + 1 + t] = mean[t];
        b[2 * H + 1 + F + t] = inv_std[t];
    }
}

// Launches the batch's passes and its gradients: into G, or one Adam step of A when G is NULL.
void launch_step(const float *params, const float *features, const float *targets, int batch, float *scratch,
                 float *G, const AdamArgs &A, float *loss, cudaStream_t s) {
    float *H1 = scratch, *H2 = H1 + size_t(batch) * H, *dH1 = H2 + size_t(batch) * H;
    float *dH2 = dH1 + size_t(batch) * H, *dO = dH2 + size_t(batch) * H;
    const int threads = 256;
    const int blocks = std::min(1184, (batch * 32 + threads - 1) / threads);
    cudaMemsetAsync(loss, 0, sizeof(float), s);
    mlp_fwd_bwd<<<blocks, threads, SMEM_FLOATS * sizeof(float), s>>>(params, features, targets,
                                                                       batch, H1, H2, dH1, dH2, dO, loss);
    // Stages for the chunks that there are: a batch of one or two needs no more shared memory than the pass before
    // it, and no attribute set (gradients of 64 samples 17.2 -> 14.1 us a call).
    const int chunks = (batch + GRAD_CHUNK - 1) / GRAD_CHUNK;
    const int smem = std::min(chunks, GRAD_STAGES) * GRAD_STAGE_FLOATS * 4;
    if (smem > 48 * 1024) cudaFuncSetAttribute(mlp_grads, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    mlp_grads<<<GRAD_BLOCKS, GRAD_THREADS, smem, s>>>(features, H1, H2, dH1, dH2, dO, batch, G, A);
}

// H1, H2, dH1, dH2 and dO (launch_step)
size_t scratch_floats(int B) { return size_t(B) * (4 * H + 1); }

}  // namespace hbm

extern "C" {

int64_t hnsw_b200_mlp_param_count(void) { return hbm::NPARAM; }

int64_t hnsw_b200_mlp_packed_bytes(void) {
    return int64_t(hbm::H * hbm::F + hbm::H * hbm::H + hbm::H) * 2 +
           int64_t(2 * hbm::H + 1 + 2 * hbm::F) * 4;
}

int64_t hnsw_b200_mlp_scratch_bytes(int32_t batch) {
    return batch < 1 ? 0 : int64_t(hbm::scratch_floats(batch) * sizeof(float));
}

int hnsw_b200_mlp_train_step(float *params, float *adam_m, float *adam_v, int64_t step, float lr,
                             const float *features, const float *targets, int32_t batch,
                             float *scratch, float *loss, void *stream) {
    using namespace hbm;
    if (!params || !adam_m || !adam_v || !features || !targets || !scratch || !loss || batch < 1 ||
        step < 1)
        return hb::fail(HNSW_B200_EINVAL, "mlp_train_step: bad argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, float(step)), c2 = 1.f - powf(b2, float(step));
    launch_step(params, features, targets, batch, scratch, nullptr,
                AdamArgs{params, adam_m, adam_v, lr, b1, b2, 1e-8f, c1, c2}, loss, s);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return hb::fail(HNSW_B200_ECUDA, std::string("mlp train: ") + cudaGetErrorString(e));
    return 0;
}

// Gradients only (no update): G receives dLoss/dparams for the batch (for gradient checks).
int hnsw_b200_mlp_gradients(const float *params, const float *features, const float *targets,
                            int32_t batch, float *scratch, float *grads, float *loss, void *stream) {
    using namespace hbm;
    if (!params || !features || !targets || !scratch || !grads || !loss || batch < 1)
        return hb::fail(HNSW_B200_EINVAL, "mlp_gradients: bad argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    launch_step(params, features, targets, batch, scratch, grads, AdamArgs{}, loss, s);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return hb::fail(HNSW_B200_ECUDA, std::string("mlp grads: ") + cudaGetErrorString(e));
    return 0;
}

int hnsw_b200_mlp_predict(const float *params, const float *features, int64_t n, float *out,
                          void *stream) {
    using namespace hbm;
    if (!params || !features || !out || n < 0) return hb::fail(HNSW_B200_EINVAL, "mlp_predict: bad argument");
    if (n == 0) return 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int threads = 256;
    const int blocks = int(std::min<int64_t>(2368, (n * 32 + threads - 1) / threads));
    mlp_predict_kernel<<<blocks, threads, SMEM_FLOATS * sizeof(float), s>>>(params, features, int(n), out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return hb::fail(HNSW_B200_ECUDA, std::string("mlp predict: ") + cudaGetErrorString(e));
    return 0;
}

int hnsw_b200_mlp_pack(const float *params, const float *mean, const float *inv_std, void *packed,
                       void *stream) {
    using namespace hbm;
    if (!params || !mean || !inv_std || !packed) return hb::fail(HNSW_B200_EINVAL, "mlp_pack: bad argument");
    mlp_pack_kernel<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        params, mean, inv_std, static_cast<unsigned char *>(packed));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return hb::fail(HNSW_B200_ECUDA, std::string("mlp pack: ") + cudaGetErrorString(e));
    return 0;
}

}  // extern "C"
