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

// Samples of a block's tile: their activations and gradients stay in shared memory.
constexpr int TS = 32;
constexpr int GRAD_THREADS = 512;  // 16 warps, two samples of a tile each
constexpr int MAX_ROWS = 296;      // blocks (rows of partial sums): two a SM
constexpr int GRAD_FLOATS = (SMEM_FLOATS + 3) / 4 * 4 + 4 * TS * H + TS * F + TS;

// Forward, backward and weight gradients of the batch: block r writes row r of part (NPARAM partial sums).
// A tile of 32 samples is run through the network a warp a sample; then every thread adds the tile's
// products to the parameters it owns (W2: 4 x 2 of its elements, read from shared memory as one 16-byte
// broadcast and one 8-byte load a sample; W1, W3, biases: up to three single ones), tile after tile in
// order, so the sums are deterministic. Bound by the shuffles and shared-memory reads of the passes,
// about 900 instructions a sample. (Writing the activations out and adding the whole batch up in
// one thread a parameter took 15 + 182 us a step of 4,096 samples; this kernel takes 20, mlp_finish 4.)
__global__ void __launch_bounds__(GRAD_THREADS) mlp_grad_tiles(const float *P, const float *X, const float *Y,
                                                               int B, float *part, float *loss) {
    extern __shared__ __align__(16) float sw[];
    float *h1 = sw + (SMEM_FLOATS + 3) / 4 * 4, *h2 = h1 + TS * H, *d1 = h2 + TS * H, *d2 = d1 + TS * H;
    float *xs = d2 + TS * H, *dos = xs + TS * F;
    load_weights(P, sw);
    const float *w2 = sw + H * S_W1 + H, *w3 = w2 + H * S_W2 + H;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int j0 = (t >> 5) * 4, i0 = (t & 31) * 2;  // W2[j0 .. j0 + 3][i0 .. i0 + 1]
    const int p1 = t, p1b = t + GRAD_THREADS;          // W1 elements
    float aw2[4][2] = {}, aw1 = 0.f, aw1b = 0.f, arest = 0.f, lsum = 0.f;
    const int tiles = (B + TS - 1) / TS;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int b0 = tile * TS, nb = min(TS, B - b0);
        for (int s = warp; s < nb; s += GRAD_THREADS / 32) {
            const int b = b0 + s;
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
            h1[s * H + lane] = h1a;
            h1[s * H + lane + 32] = h1b;
            h2[s * H + lane] = h2a;
            h2[s * H + lane + 32] = h2b;
            d1[s * H + lane] = h1a > 0.f ? g1a : 0.f;
            d1[s * H + lane + 32] = h1b > 0.f ? g1b : 0.f;
            d2[s * H + lane] = g2a;
            d2[s * H + lane + 32] = g2b;
            if (lane < F) xs[s * F + lane] = X[int64_t(b) * F + lane];
            if (lane == 0) dos[s] = g;
        }
        __syncthreads();
        // dW1 = dH1^T X, dW2 = dH2^T H1, dW3 = dO^T H2, biases the column sums
#pragma unroll 4
        for (int s = 0; s < nb; s++) {
            const float4 d = *reinterpret_cast<const float4 *>(d2 + s * H + j0);
            const float2 h = *reinterpret_cast<const float2 *>(h1 + s * H + i0);
            aw2[0][0] = fmaf(d.x, h.x, aw2[0][0]);
            aw2[0][1] = fmaf(d.x, h.y, aw2[0][1]);
            aw2[1][0] = fmaf(d.y, h.x, aw2[1][0]);
            aw2[1][1] = fmaf(d.y, h.y, aw2[1][1]);
            aw2[2][0] = fmaf(d.z, h.x, aw2[2][0]);
            aw2[2][1] = fmaf(d.z, h.y, aw2[2][1]);
            aw2[3][0] = fmaf(d.w, h.x, aw2[3][0]);
            aw2[3][1] = fmaf(d.w, h.y, aw2[3][1]);
        }
        for (int s = 0; s < nb; s++) {
            aw1 = fmaf(d1[s * H + p1 / F], xs[s * F + p1 % F], aw1);
            if (p1b < H * F) aw1b = fmaf(d1[s * H + p1b / F], xs[s * F + p1b % F], aw1b);
            if (t < H) arest += d1[s * H + t];
            else if (t < 2 * H) arest += d2[s * H + t - H];
            else if (t < 3 * H) arest = fmaf(dos[s], h2[s * H + t - 2 * H], arest);
            else if (t == 3 * H) arest += dos[s];
        }
        __syncthreads();  // before the next tile's samples are written
    }
    float *row = part + int64_t(blockIdx.x) * NPARAM;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        row[O_W2 + (j0 + a) * H + i0] = aw2[a][0];
        row[O_W2 + (j0 + a) * H + i0 + 1] = aw2[a][1];
    }
    row[O_W1 + p1] = aw1;
    if (p1b < H * F) row[O_W1 + p1b] = aw1b;
    if (t < H) row[O_B1 + t] = arest;
    else if (t < 2 * H) row[O_B2 + t - H] = arest;
    else if (t < 3 * H) row[O_W3 + t - 2 * H] = arest;
    else if (t == 3 * H) row[O_B3] = arest;
    if (lane == 0 && lsum != 0.f) atomicAdd(loss, lsum);
}

// A parameter's gradient: the rows of partial sums added up in a fixed order, four threads a parameter
// (rows 0, 4, 8, ...; 1, 5, ...; then the four sums). G != NULL: written there. Else one Adam step
// (Kingma & Ba) with bias correction on the float32 masters.
constexpr int FIN_PARAMS = 64;
__global__ void mlp_finish(const float *part, int rows, float *G, float *P, float *M, float *V, float lr, float b1,
                           float b2, float eps, float c1, float c2) {
    __shared__ float sums[4][FIN_PARAMS];
    const int i = threadIdx.x % FIN_PARAMS, q = threadIdx.x / FIN_PARAMS;
    const int p = blockIdx.x * FIN_PARAMS + i;
    float acc = 0.f;
    if (p < NPARAM) {
#pragma unroll 8
        for (int r = q; r < rows; r += 4) acc += part[int64_t(r) * NPARAM + p];
    }
    sums[q][i] = acc;
    __syncthreads();
    if (q != 0 || p >= NPARAM) return;
    const float g = (sums[0][i] + sums[1][i]) + (sums[2][i] + sums[3][i]);
    if (G) {
        G[p] = g;
        return;
    }
    const float m = b1 * M[p] + (1.f - b1) * g;
    const float v = b2 * V[p] + (1.f - b2) * g * g;
    M[p] = m;
    V[p] = v;
    P[p] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
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

size_t scratch_floats(int B) { return size_t(B) * (4 * H + 1) + NPARAM + 4; }  // at least the partial sums

// Launches the batch's gradients into rows of part (scratch), and returns how many rows.
int grad_rows(const float *params, const float *features, const float *targets, int batch, float *part,
              float *loss, cudaStream_t s) {
    const int rows = std::min(MAX_ROWS, (batch + TS - 1) / TS);
    cudaFuncSetAttribute(mlp_grad_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, GRAD_FLOATS * 4);
    cudaMemsetAsync(loss, 0, sizeof(float), s);
    mlp_grad_tiles<<<rows, GRAD_THREADS, GRAD_FLOATS * sizeof(float), s>>>(params, features, targets, batch, part,
                                                                            loss);
    return rows;
}

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
    const int rows = grad_rows(params, features, targets, batch, scratch, loss, s);
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, float(step)), c2 = 1.f - powf(b2, float(step));
    mlp_finish<<<(NPARAM + FIN_PARAMS - 1) / FIN_PARAMS, 4 * FIN_PARAMS, 0, s>>>(
        scratch, rows, nullptr, params, adam_m, adam_v, lr, b1, b2, 1e-8f, c1, c2);
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
    const int rows = grad_rows(params, features, targets, batch, scratch, loss, s);
    mlp_finish<<<(NPARAM + FIN_PARAMS - 1) / FIN_PARAMS, 4 * FIN_PARAMS, 0, s>>>(
        scratch, rows, grads, nullptr, nullptr, nullptr, 0.f, 0.f, 0.f, 0.f, 1.f, 1.f);
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
