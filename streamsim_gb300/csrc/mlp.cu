// mlp.cu — the warm-start network: MLP 12 -> 128 -> 128 -> 64, GELU,
// BF16 weights with an FP32 master copy, FP32 accumulation, trained by the
// library's own forward, backward and Adam kernels.
//
// Layout: parameters are one FP32 vector (W1[128x12], b1[128], W2[128x128],
// b2[128], W3[64x128], b3[64], row-major, W[out][in]); a BF16 copy of the
// weights is what the forward and backward GEMMs read.  Activations are
// row-major [n][features] FP32.  The loss is the mean squared error over
// all n x 64 outputs.
//
// GEMMs (FP32 FMA: activations and gradients are FP32, and so are the sums).
//   k_layer  128 rows per CTA against a whole weight matrix in shared memory
//            (at most 128 x 128 floats), 8 x 8 or 8 x 4 outputs per thread;
//            the epilogue is the layer's own: bias and GELU, bias and loss,
//            or the product with GELU'(Z)
//   k_wgrad  a weight gradient dZ^T A over a share of the rows per CTA, with
//            the bias gradient beside it; every CTA writes its own partial
//            and k_sum_partials adds them in a fixed order, so a training
//            step is deterministic.
#include <cuda_bf16.h>

#include <cmath>

#include "internal.h"

namespace facetcu {
namespace mlp {


namespace {

__device__ __forceinline__ float gelu(float z)
{
    return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad(float z)
{
    const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

// acc[i][j] += a[i] * b[j], two columns at a time (fma.rn.f32x2: each half is
// an fma of its own).
__device__ __forceinline__ void fma2(float& c0, float& c1, float a, float b0, float b1)
{
    asm("{ .reg .b64 c, x, y;\n  mov.b64 c, {%0, %1};\n  mov.b64 x, {%2, %2};\n"
        "  mov.b64 y, {%3, %4};\n  fma.rn.f32x2 c, x, y, c;\n  mov.b64 {%0, %1}, c; }"
        : "+f"(c0), "+f"(c1)
        : "f"(a), "f"(b0), "f"(b1));
}

// ---- layers -------------------------------------------------------------------
enum Epilogue {
    kGelu,      // Z = acc + bias to out (where given), GELU(Z) to out2
    kOutput,    // acc + bias to out
    kLoss,      // Y = acc + bias; out = 2 (Y - T) scale, the CTA's sum of (Y - T)^2
    kGeluBack,  // acc * GELU'(Z)
};
struct LayerArgs {
    const float* bias;
    const float* other;  // kLoss: the targets T; kGeluBack: Z
    float *out, *out2;
    double* loss_part;
    float scale;
};

constexpr int kRows = 128;      // rows of a CTA
constexpr int kPad = kRows + 4;

// Bound: FP32 FMA issue and, in the epilogues, erf and exp.  The layers of a
// 65,536-row gradient take 243 us and the weight gradients 95 (10.3 GFLOP: 31
// TFLOP/s over both); with 64 x 64 tiles, 4 x 4 outputs per thread, separate
// loss, GELU and bias kernels they took 1,440, and a one-thread sum of the loss
// 963 more.
// out[rows][N] = A[rows][K] B, B = W^T (kT: W is [N][K]) or W ([K][N]), in K
// slices of KS whose A values are fetched while the slice before is summed.
template <int K, int N, int KS, bool kT, Epilogue E>
__global__ void __launch_bounds__(256, 2) k_layer(int rows, const float* __restrict__ A,
                                                  const __nv_bfloat16* __restrict__ W,
                                                  LayerArgs args)
{
    static_assert(K % KS == 0 && KS % 4 == 0 && (N == 128 || N == 64), "shape");
    constexpr int C = N / 16;                          // columns per thread
    constexpr int kQuads = kRows * KS / 4;             // float4 of a slice
    constexpr int kFetch = (kQuads + 255) / 256;
    extern __shared__ __align__(16) float smem[];
    float(*Bs)[N] = reinterpret_cast<float(*)[N]>(smem);                 // [K][N]
    float(*As)[KS][kPad] = reinterpret_cast<float(*)[KS][kPad]>(smem + K * N);  // [2][KS][rows]
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    if (kT) {  // lanes over n: the stores of a warp are side by side
        constexpr int V = K % 8 == 0 ? 8 : 4;  // weights per load
        for (int i = threadIdx.x; i < K / V * N; i += 256) {
            const int n = i % N, k = i / N * V;
            __nv_bfloat16 w[V];
            if (V == 8) *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(W + n * K + k);
            else *reinterpret_cast<uint2*>(w) = *reinterpret_cast<const uint2*>(W + n * K + k);
#pragma unroll
            for (int j = 0; j < V; ++j) Bs[k + j][n] = __bfloat162float(w[j]);
        }
    } else {
        for (int i = threadIdx.x; i < K * N; i += 256) Bs[i / N][i % N] = __bfloat162float(W[i]);
    }
    double loss = 0.0;
    for (int r0 = blockIdx.x * kRows; r0 < rows; r0 += gridDim.x * kRows) {
    float4 next[kFetch];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < kFetch; ++q) {
            const int i = threadIdx.x + q * 256, r = i / (KS / 4), k = i % (KS / 4) * 4;
            next[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if ((kQuads % 256 == 0 || i < kQuads) && r0 + r < rows)
                next[q] = *reinterpret_cast<const float4*>(A + size_t(r0 + r) * K + k0 + k);
        }
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int q = 0; q < kFetch; ++q) {
            const int i = threadIdx.x + q * 256, r = i / (KS / 4), k = i % (KS / 4) * 4;
            if (kQuads % 256 == 0 || i < kQuads) {
                As[buf][k][r] = next[q].x;
                As[buf][k + 1][r] = next[q].y;
                As[buf][k + 2][r] = next[q].z;
                As[buf][k + 3][r] = next[q].w;
            }
        }
    };
    float acc[8][C] = {};
    fetch(0);
    put(0);
    __syncthreads();
#pragma unroll 1
    for (int k0 = 0, buf = 0; k0 < K; k0 += KS, buf ^= 1) {
        if (k0 + KS < K) fetch(k0 + KS);
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            float a[8], b[C];
            // rows 4 ty .. and 64 + 4 ty .., columns 4 tx .. and 64 + 4 tx ..
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&As[buf][k][4 * ty]);
            *reinterpret_cast<float4*>(a + 4) =
                *reinterpret_cast<const float4*>(&As[buf][k][64 + 4 * ty]);
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&Bs[k0 + k][4 * tx]);
            if (C == 8)
                *reinterpret_cast<float4*>(b + C - 4) =
                    *reinterpret_cast<const float4*>(&Bs[k0 + k][N - 64 + 4 * tx]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < C; j += 2)
                    fma2(acc[i][j], acc[i][j + 1], a[i], b[j], b[j + 1]);
        }
        if (k0 + KS < K) put(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = r0 + (i < 4 ? 0 : 64) + 4 * ty + i % 4;
        if (r >= rows) continue;
#pragma unroll
        for (int h = 0; h < C / 4; ++h) {
            const int n = h * 64 + 4 * tx;
            const size_t at = size_t(r) * N + n;
            float v[4], w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = acc[i][h * 4 + j];
            if (E != kGeluBack) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += args.bias[n + j];
            }
            if (E == kLoss || E == kGeluBack)
                *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(args.other + at);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (E == kGelu) w[j] = gelu(v[j]);
                if (E == kGeluBack) v[j] *= gelu_grad(w[j]);
                if (E == kLoss) {
                    const float d = v[j] - w[j];
                    loss += double(d) * double(d);
                    v[j] = 2.0f * d * args.scale;
                }
            }
            if (E != kGelu || args.out)
                *reinterpret_cast<float4*>(args.out + at) = make_float4(v[0], v[1], v[2], v[3]);
            if (E == kGelu)
                *reinterpret_cast<float4*>(args.out2 + at) = make_float4(w[0], w[1], w[2], w[3]);
        }
    }
    }
    if (E == kLoss) {
        double* red = reinterpret_cast<double*>(smem);  // (the operands are done with)
        red[threadIdx.x] = loss;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) args.loss_part[blockIdx.x] = red[0];
    }
}

// CTAs of a layer: two per SM, each loads the weights once.
inline int layer_ctas(int rows)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::min((rows + kRows - 1) / kRows, 2 * std::max(sms, 1));
}

template <int K, int N, int KS, bool kT, Epilogue E>
void layer(int rows, const float* A, const __nv_bfloat16* W, const LayerArgs& args, cudaStream_t s)
{
    constexpr int smem = (K * N + 2 * KS * kPad) * 4;
    FCU_CHECK(cudaFuncSetAttribute(k_layer<K, N, KS, kT, E>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_layer<K, N, KS, kT, E><<<layer_ctas(rows), 256, smem, s>>>(rows, A, W, args);
    FCU_LAUNCH("k_layer");
}

// ---- weight gradients ---------------------------------------------------------
constexpr int kSlice = 16;  // rows in shared memory at a time

// part[cta][o * I + i] = sum of D[r][o] X[r][i] over the CTA's rows, and
// bias_part[cta][o] = sum of D[r][o]; `stride` floats from one CTA's partials to
// the next's.  I = 128: 8 x 8 (O = 128) or 4 x 8 (O = 64) outputs per thread.
template <int O>
__global__ void __launch_bounds__(256, 2) k_wgrad(int rows, int rows_per_cta,
                                                  const float* __restrict__ D,
                                                  const float* __restrict__ X, size_t stride,
                                                  float* __restrict__ part,
                                                  float* __restrict__ bias_part)
{
    constexpr int I = 128, R = O / 16;
    __shared__ __align__(16) float Ds[2][kSlice][O];
    __shared__ __align__(16) float Xs[2][kSlice][I];
    constexpr int kFd = kSlice * O / 4 / 256, kFx = kSlice * I / 4 / 256;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int begin = blockIdx.x * rows_per_cta, end = min(rows, begin + rows_per_cta);
    float4 nd[kFd], nx[kFx];
    auto fetch = [&](int r0) {
#pragma unroll
        for (int q = 0; q < kFd; ++q) {
            const int i = threadIdx.x + q * 256, r = r0 + i / (O / 4);
            nd[q] = r < end ? reinterpret_cast<const float4*>(D + size_t(r) * O)[i % (O / 4)]
                            : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int q = 0; q < kFx; ++q) {
            const int i = threadIdx.x + q * 256, r = r0 + i / (I / 4);
            nx[q] = r < end ? reinterpret_cast<const float4*>(X + size_t(r) * I)[i % (I / 4)]
                            : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int q = 0; q < kFd; ++q) reinterpret_cast<float4*>(Ds[buf])[threadIdx.x + q * 256] = nd[q];
#pragma unroll
        for (int q = 0; q < kFx; ++q) reinterpret_cast<float4*>(Xs[buf])[threadIdx.x + q * 256] = nx[q];
    };
    float acc[R][8] = {}, bias = 0.0f;
    fetch(begin);
    put(0);
    __syncthreads();
#pragma unroll 1
    for (int r0 = begin, buf = 0; r0 < end; r0 += kSlice, buf ^= 1) {
        if (r0 + kSlice < end) fetch(r0 + kSlice);
#pragma unroll
        for (int k = 0; k < kSlice; ++k) {
            float a[R], b[8];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&Ds[buf][k][4 * ty]);
            if (R == 8)
                *reinterpret_cast<float4*>(a + R - 4) =
                    *reinterpret_cast<const float4*>(&Ds[buf][k][O - 64 + 4 * ty]);
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&Xs[buf][k][4 * tx]);
            *reinterpret_cast<float4*>(b + 4) =
                *reinterpret_cast<const float4*>(&Xs[buf][k][64 + 4 * tx]);
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < 8; j += 2)
                    fma2(acc[i][j], acc[i][j + 1], a[i], b[j], b[j + 1]);
        }
        if (threadIdx.x < O) {
#pragma unroll
            for (int k = 0; k < kSlice; ++k) bias += Ds[buf][k][threadIdx.x];
        }
        if (r0 + kSlice < end) put(buf ^ 1);
        __syncthreads();
    }
    float* p = part + size_t(blockIdx.x) * stride;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int o = (i < 4 ? 0 : 64) + 4 * ty + i % 4;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<float4*>(p + o * I + h * 64 + 4 * tx) = make_float4(
                acc[i][h * 4], acc[i][h * 4 + 1], acc[i][h * 4 + 2], acc[i][h * 4 + 3]);
    }
    if (threadIdx.x < O) bias_part[size_t(blockIdx.x) * stride + threadIdx.x] = bias;
}

// The first layer's gradient (I = 12 inputs): thread (o, half) sums 6 of a
// weight row's 12 outputs.
__global__ void __launch_bounds__(256) k_wgrad_first(int rows, int rows_per_cta,
                                                     const float* __restrict__ D,
                                                     const float* __restrict__ X, size_t stride,
                                                     float* __restrict__ part,
                                                     float* __restrict__ bias_part)
{
    constexpr int kTake = 64, U = 16;  // rows of X kept, rows of D in flight
    __shared__ __align__(16) float Xs[kTake][kIn];
    const int o = threadIdx.x % kH, half = threadIdx.x / kH;
    const int begin = blockIdx.x * rows_per_cta, end = min(rows, begin + rows_per_cta);
    float acc[6] = {}, bias = 0.0f;
    for (int r0 = begin; r0 < end; r0 += kTake) {
        const int n = min(kTake, end - r0);
        __syncthreads();
        for (int i = threadIdx.x; i < n * kIn; i += 256) (&Xs[0][0])[i] = X[size_t(r0) * kIn + i];
        __syncthreads();
        for (int k = 0; k < n; k += U) {
            float d[U];
#pragma unroll
            for (int u = 0; u < U; ++u) d[u] = k + u < n ? D[size_t(r0 + k + u) * kH + o] : 0.0f;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u >= n) break;
                bias += d[u];
#pragma unroll
                for (int j = 0; j < 6; ++j) acc[j] += d[u] * Xs[k + u][half * 6 + j];
            }
        }
    }
    float* p = part + size_t(blockIdx.x) * stride;
#pragma unroll
    for (int j = 0; j < 6; ++j) p[o * kIn + half * 6 + j] = acc[j];
    if (half == 0) bias_part[size_t(blockIdx.x) * stride + o] = bias;
}

// out[i] = sum over the CTAs' partials, in order within each of 8 interleaved
// runs and then over the runs.
__global__ void __launch_bounds__(256) k_sum_partials(const float* __restrict__ part, int ctas,
                                                      int n, float* __restrict__ out)
{
    __shared__ float red[8][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), run = threadIdx.x >> 5;
    float s = 0.0f;
    if (i < n)
        for (int z = run; z < ctas; z += 8) s += part[size_t(z) * n + i];
    red[run][threadIdx.x & 31] = s;
    __syncthreads();
    if (run == 0 && i < n) {
        for (int k = 1; k < 8; ++k) s += red[k][threadIdx.x];
        out[i] = s;
    }
}

__global__ void __launch_bounds__(256) k_sum_double(const double* part, int n, double* out)
{
    __shared__ double red[256];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += 256) s += part[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

__global__ void k_to_bf16(const float* p, size_t n, __nv_bfloat16* q)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) q[i] = __float2bfloat16_rn(p[i]);
}

// Adam (Kingma & Ba 2015) with bias correction.
__global__ void k_adam(float* p, const float* g, float* m, float* v, size_t n, float lr, float b1,
                       float b2, float eps, float c1, float c2)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// Gather a minibatch: rows idx[i] of X (cols c) into out.
__global__ void k_gather_rows(const float* X, const uint32_t* idx, int n, int cols, float* out)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= size_t(n) * cols) return;
    const size_t r = i / cols, c = i % cols;
    out[i] = X[size_t(idx[r]) * cols + c];
}

// Minibatch indices from a counter-based hash (splitmix64 of seed, step, i).
__global__ void k_batch_indices(uint64_t seed, uint64_t step, int n, uint64_t population,
                                uint32_t* idx)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (step * 0x100000001ull + uint64_t(i) + 1ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    idx[i] = uint32_t(z % population);
}

inline unsigned blocks(size_t n, unsigned b) { return unsigned((n + b - 1) / b); }

}  // namespace

// ---- host side ---------------------------------------------------------------
static_assert(kParams == kParameterCount, "parameter layout");

void init_params(Net& net, uint32_t seed, cudaStream_t s)
{
    // Glorot-uniform weights, zero biases, from a host RNG (xorshift64*).
    std::vector<float> p(kParams, 0.0f);
    uint64_t state = 0x2545F4914F6CDD1Dull ^ (uint64_t(seed) * 0x9E3779B97F4A7C15ull);
    auto uni = [&]() {
        state ^= state >> 12;
        state ^= state << 25;
        state ^= state >> 27;
        const uint64_t r = state * 2685821657736338717ull;
        return double(r >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int fan_out, int fan_in) {
        const double lim = std::sqrt(6.0 / double(fan_in + fan_out));
        for (int i = 0; i < fan_out * fan_in; ++i) p[off + i] = float((2.0 * uni() - 1.0) * lim);
    };
    fill(kOffW1, kH, kIn);
    fill(kOffW2, kH, kH);
    fill(kOffW3, kOut, kH);
    net.params.reserve(kParams * 4);
    FCU_CHECK(cudaMemcpyAsync(net.params.ptr, p.data(), kParams * 4, cudaMemcpyHostToDevice, s));
    net.adam_m.reserve(kParams * 4);
    net.adam_v.reserve(kParams * 4);
    net.grad.reserve(kParams * 4);
    FCU_CHECK(cudaMemsetAsync(net.adam_m.ptr, 0, kParams * 4, s));
    FCU_CHECK(cudaMemsetAsync(net.adam_v.ptr, 0, kParams * 4, s));
    net.bf16.reserve(kParams * 2);
    k_to_bf16<<<blocks(kParams, 256), 256, 0, s>>>(net.params.as<float>(), kParams,
                                                   net.bf16.as<__nv_bfloat16>());
    FCU_LAUNCH("k_to_bf16");
    net.ready = true;
    net.steps_done = 0;
}

void set_params(Net& net, const float* host, cudaStream_t s)
{
    if (!net.ready) init_params(net, 1, s);
    FCU_CHECK(cudaMemcpyAsync(net.params.ptr, host, kParams * 4, cudaMemcpyHostToDevice, s));
    FCU_CHECK(cudaMemsetAsync(net.adam_m.ptr, 0, kParams * 4, s));
    FCU_CHECK(cudaMemsetAsync(net.adam_v.ptr, 0, kParams * 4, s));
    k_to_bf16<<<blocks(kParams, 256), 256, 0, s>>>(net.params.as<float>(), kParams,
                                                   net.bf16.as<__nv_bfloat16>());
    FCU_LAUNCH("k_to_bf16");
    net.steps_done = 0;
}

// The hidden layers of n rows: GELU(Z) to sc.a1, sc.a2 and, for a backward
// pass, Z to sc.z1, sc.z2.
static void hidden(Net& net, const float* X, int n, Scratch& sc, bool keep_z, cudaStream_t s)
{
    const __nv_bfloat16* w = net.bf16.as<__nv_bfloat16>();
    const float* p = net.params.as<float>();
    float* z1 = keep_z ? static_cast<float*>(sc.z1.reserve(size_t(n) * kH * 4)) : nullptr;
    float* a1 = static_cast<float*>(sc.a1.reserve(size_t(n) * kH * 4));
    float* z2 = keep_z ? static_cast<float*>(sc.z2.reserve(size_t(n) * kH * 4)) : nullptr;
    float* a2 = static_cast<float*>(sc.a2.reserve(size_t(n) * kH * 4));
    layer<kIn, kH, kIn, true, kGelu>(n, X, w + kOffW1, {p + kOffB1, nullptr, z1, a1, nullptr, 0.0f}, s);
    layer<kH, kH, 16, true, kGelu>(n, a1, w + kOffW2, {p + kOffB2, nullptr, z2, a2, nullptr, 0.0f}, s);
}

void forward_full(Net& net, const float* X, int n, Scratch& sc, float* Y, cudaStream_t s)
{
    hidden(net, X, n, sc, false, s);
    layer<kH, kOut, 16, true, kOutput>(n, sc.a2.as<float>(), net.bf16.as<__nv_bfloat16>() + kOffW3,
                                       {net.params.as<float>() + kOffB3, nullptr, Y, nullptr,
                                        nullptr, 0.0f},
                                       s);
}

// Inference over any number of rows: chunks of kInferChunk rows keep the
// activation scratch at 1 GB and the GEMM grid within its y limit.
void infer(Net& net, const float* X, size_t n, Scratch& sc, float* Y, cudaStream_t s)
{
    for (size_t r0 = 0; r0 < n; r0 += kInferChunk) {
        const int rows = int(std::min(n - r0, kInferChunk));
        forward_full(net, X + r0 * kIn, rows, sc, Y + r0 * kOut, s);
    }
}

// Loss and gradient (into net.grad) of one batch; returns the mean loss.
double loss_and_grad(Net& net, const float* X, const float* T, int n, Scratch& sc, cudaStream_t s,
                     bool want_loss)
{
    const __nv_bfloat16* w = net.bf16.as<__nv_bfloat16>();
    const float* p = net.params.as<float>();
    hidden(net, X, n, sc, true, s);
    const float *z1 = sc.z1.as<float>(), *a1 = sc.a1.as<float>(), *z2 = sc.z2.as<float>(),
                *a2 = sc.a2.as<float>();
    float* dy = static_cast<float*>(sc.dy.reserve(size_t(n) * kOut * 4));
    float* dz2 = static_cast<float*>(sc.da.reserve(size_t(n) * kH * 4));
    float* dz1 = static_cast<float*>(sc.dz.reserve(size_t(n) * kH * 4));
    const size_t cnt = size_t(n) * kOut;
    const int tiles = layer_ctas(n);
    double* lossp = static_cast<double*>(sc.lossp.reserve((size_t(tiles) + 1) * 8));
    layer<kH, kOut, 16, true, kLoss>(n, a2, w + kOffW3,
                                     {p + kOffB3, T, dy, nullptr, lossp, 1.0f / float(cnt)}, s);
    // dZ2 = dY W3 gelu'(Z2) ; dZ1 = dZ2 W2 gelu'(Z1)
    layer<kOut, kH, 16, false, kGeluBack>(n, dy, w + kOffW3, {nullptr, z2, dz2, nullptr, nullptr, 0.0f}, s);
    layer<kH, kH, 16, false, kGeluBack>(n, dz2, w + kOffW2, {nullptr, z1, dz1, nullptr, nullptr, 0.0f}, s);
    // weight and bias gradients: two CTAs per SM, at least 64 rows each
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int want = std::max(1, std::min(2 * std::max(sms, 1), n / 64));
    const int per = (n + want - 1) / want;
    const int ctas = (n + per - 1) / per;
    float* part = static_cast<float*>(sc.part.reserve(size_t(ctas) * kParams * 4));
    k_wgrad<kOut><<<ctas, 256, 0, s>>>(n, per, dy, a2, kParams, part + kOffW3, part + kOffB3);
    k_wgrad<kH><<<ctas, 256, 0, s>>>(n, per, dz2, a1, kParams, part + kOffW2, part + kOffB2);
    k_wgrad_first<<<ctas, 256, 0, s>>>(n, per, dz1, X, kParams, part + kOffW1, part + kOffB1);
    k_sum_partials<<<blocks(kParams, 32), 256, 0, s>>>(part, ctas, kParams, net.grad.as<float>());
    FCU_LAUNCH("mlp backward");
    if (!want_loss) return 0.0;
    double* total = lossp + tiles;
    k_sum_double<<<1, 256, 0, s>>>(lossp, tiles, total);
    double host = 0.0;
    FCU_CHECK(cudaMemcpyAsync(&host, total, 8, cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaStreamSynchronize(s));
    return host / double(cnt);
}

void adam_step(Net& net, float lr, cudaStream_t s)
{
    net.steps_done += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, float(net.steps_done));
    const float c2 = 1.0f - std::pow(b2, float(net.steps_done));
    k_adam<<<blocks(kParams, 256), 256, 0, s>>>(net.params.as<float>(), net.grad.as<float>(),
                                                net.adam_m.as<float>(), net.adam_v.as<float>(),
                                                kParams, lr, b1, b2, 1e-8f, c1, c2);
    FCU_LAUNCH("k_adam");
    k_to_bf16<<<blocks(kParams, 256), 256, 0, s>>>(net.params.as<float>(), kParams,
                                                   net.bf16.as<__nv_bfloat16>());
    FCU_LAUNCH("k_to_bf16");
}

// Train on n samples resident on the device (X[n][12], T[n][64]).
double train(Net& net, const float* X, const float* T, uint64_t n, uint32_t steps, uint32_t batch,
             float lr, uint32_t seed, Scratch& sc, cudaStream_t s)
{
    uint32_t* idx = static_cast<uint32_t*>(sc.idx.reserve(size_t(batch) * 4));
    float* xb = static_cast<float*>(sc.xb.reserve(size_t(batch) * kIn * 4));
    float* tb = static_cast<float*>(sc.tb.reserve(size_t(batch) * kOut * 4));
    double last = 0.0;
    for (uint32_t st = 0; st < steps; ++st) {
        k_batch_indices<<<blocks(batch, 256), 256, 0, s>>>(seed, st, int(batch), n, idx);
        k_gather_rows<<<blocks(size_t(batch) * kIn, 256), 256, 0, s>>>(X, idx, int(batch), kIn, xb);
        k_gather_rows<<<blocks(size_t(batch) * kOut, 256), 256, 0, s>>>(T, idx, int(batch), kOut, tb);
        const bool report = st + 1 == steps;
        const double l = loss_and_grad(net, xb, tb, int(batch), sc, s, report);
        if (report) last = l;
        adam_step(net, lr, s);
    }
    FCU_CHECK(cudaStreamSynchronize(s));
    return last;
}

// ---- features and warm start ----------------------------------------------
// Per (sun k, side s): the first-order radiosity B1 (one sweep from zero) of
// 8 band groups (bands 0, 9, ..., 63) scaled by ref_b = sky_b + beam_b, the
// reflectance and transmittance of band 32, the sky-view fraction
// sky_s / denom_s (1 when denom = 0) and the side normal's y (up) component.
__global__ void k_features(const float* B1, uint32_t S, uint32_t bands, uint32_t suns,
                           const float* rho, const float* tau, const float* sky,
                           const float* beam, const uint32_t* denom, const uint32_t* skyc,
                           const facetcu_vertex* V, float* X)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= size_t(S) * suns) return;
    const uint32_t k = uint32_t(i / S), s = uint32_t(i % S);
    float* x = X + i * kIn;
    for (int g = 0; g < 8; ++g) {
        const uint32_t b = uint32_t(g * 9);
        const float ref = sky[b] + beam[b];
        x[g] = B1[(size_t(k) * bands + b) * S + s] / (ref > 0.0f ? ref : 1.0f);
    }
    const uint32_t mid = bands / 2;
    x[8] = rho[size_t(mid) * S + s];
    x[9] = tau[size_t(mid) * S + s];
    x[10] = denom[s] ? float(skyc[s]) / float(denom[s]) : 1.0f;
    const float ny = V[3 * (s >> 1)].normal[1];
    x[11] = (s & 1u) ? -ny : ny;
}

// x0[k*bands + b][s] = B1 + Y[(k*S + s)][b] * ref_b  (Y = predicted (B - B1) / ref)
__global__ void k_warm_combine(const float* B1, const float* Y, uint32_t S, uint32_t bands,
                               uint32_t suns, const float* sky, const float* beam, float* x0)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t total = size_t(S) * bands * suns;
    if (i >= total) return;
    const size_t col = i / S;
    const uint32_t s = uint32_t(i % S);
    const uint32_t b = uint32_t(col % bands), k = uint32_t(col / bands);
    const float ref = sky[b] + beam[b];
    const float y = Y[(size_t(k) * S + s) * kOut + b];
    x0[i] = fmaxf(0.0f, B1[i] + y * ref);
}

// T[(k*S + s)][b] = (B - B1) / ref_b  (training targets)
__global__ void k_targets(const float* B, const float* B1, uint32_t S, uint32_t bands,
                          uint32_t suns, const float* sky, const float* beam, float* T)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t total = size_t(S) * bands * suns;
    if (i >= total) return;
    const size_t col = i / S;
    const uint32_t s = uint32_t(i % S);
    const uint32_t b = uint32_t(col % bands), k = uint32_t(col / bands);
    const float ref = sky[b] + beam[b];
    T[(size_t(k) * S + s) * kOut + b] = (B[i] - B1[i]) / (ref > 0.0f ? ref : 1.0f);
}

void features(const float* B1, uint32_t S, uint32_t bands, uint32_t suns, const float* rho,
              const float* tau, const float* sky, const float* beam, const uint32_t* denom,
              const uint32_t* skyc, const facetcu_vertex* V, float* X, cudaStream_t s)
{
    k_features<<<blocks(size_t(S) * suns, 256), 256, 0, s>>>(B1, S, bands, suns, rho, tau, sky,
                                                             beam, denom, skyc, V, X);
    FCU_LAUNCH("k_features");
}

void warm_combine(const float* B1, const float* Y, uint32_t S, uint32_t bands, uint32_t suns,
                  const float* sky, const float* beam, float* x0, cudaStream_t s)
{
    k_warm_combine<<<blocks(size_t(S) * bands * suns, 256), 256, 0, s>>>(B1, Y, S, bands, suns,
                                                                         sky, beam, x0);
    FCU_LAUNCH("k_warm_combine");
}

void targets(const float* B, const float* B1, uint32_t S, uint32_t bands, uint32_t suns,
             const float* sky, const float* beam, float* T, cudaStream_t s)
{
    k_targets<<<blocks(size_t(S) * bands * suns, 256), 256, 0, s>>>(B, B1, S, bands, suns, sky,
                                                                    beam, T);
    FCU_LAUNCH("k_targets");
}

}  // namespace mlp
}  // namespace facetcu
