// solve.cu — the reference's single-RHS Jacobi sweep and incident irradiance.
//
// k_jacobi_rows is the sweep of the reference's radiosity.comp:49-106
// (FacetrtVulkan::solve): FP32 gather over the count-form CSR, both sides of a
// facet updated together, mix() relaxation, max|dB| as an atomicMax over float
// bits.  It serves the graphs that column.cu's plan is not made for (few
// edges, short rows); k_jacobi_any is the same for callers that bring their own
// arrays.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "internal.h"

namespace facetcu {
namespace {

// The side of a thread where L of a block's 256 threads take one.  (As (256 block +
// thread) / L it wrapped at 2^30 sides of four lanes.)
constexpr __host__ __device__ uint32_t side_of(uint32_t block, uint32_t thread, uint32_t L)
{
    return block * (256u / L) + thread / L;
}
// the last side of 2^30 facets, the most that setGeometry takes
static_assert(side_of((1u << 31) / 64u - 1u, 255u, 4u) == (1u << 31) - 1u, "4 lanes");

// L lanes per side, so a facet's two rows are read at once by 2 L lanes:
// each lane has U edges in flight and the chain of dependent loads of a row
// (offsets, edge words, neighbour values) is paid once for all of them.
// (One thread per facet walked ~30 such chains: 7.2 us per sweep on the
// 4,096-facet scene of 98,000 edges, 4.1 here, 2.9 where a sweep begins while
// the one before it ends: 64 sweeps 333 -> 243 us, of 1.3 M edges 669 -> 521.)
// L follows the mean row length (lanes_for).
// kEarly: launched while the sweep before it ends; only what that one writes is
// waited for.  (With optics read after the wait, so that any kernel might write
// them, 64 sweeps of the 4,096-facet scene took 1.3 % longer.)
struct SideRow {
    uint32_t start, end, denom, skyc;  // skyc and optics in the row's first lane
    facetcu_surface_optics optics;
};
template <int L>
__device__ __forceinline__ SideRow load_row(
    bool valid, uint32_t s, const uint32_t* __restrict__ rows, const uint32_t* __restrict__ denom,
    const uint32_t* __restrict__ skyc, const facetcu_surface_optics* __restrict__ optics)
{
    SideRow r{};
    if (valid) {
        r.start = rows[s];
        r.end = rows[s + 1];
        r.denom = denom[s];
        if (threadIdx.x % L == 0) {
            r.skyc = skyc[s];
            r.optics = optics[s];
        }
    }
    return r;
}
// The new value of side s by its L lanes (whole warps, for the shuffles); returns
// |dB| in the first of them.
template <int L>
__device__ __forceinline__ float sweep_row(bool valid, uint32_t s, const SideRow& r,
                                           const facetcu_csr_edge* __restrict__ edges, float sky,
                                           float relax, const float* Bin, float* Bout)
{
    constexpr int U = 4;
    const uint32_t eg = threadIdx.x % L;
    float acc = 0.0f, old = 0.0f;
    if (valid) {
        if (eg == 0) old = Bin[s];
        for (uint32_t e = r.start + eg; e < r.end; e += L * U) {
            facetcu_csr_edge ed[U];
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ed[u] = {0u, 0u};
                if (e + u * L < r.end) ed[u] = edges[e + u * L];
            }
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = e + u * L < r.end ? Bin[ed[u].neighbor] : 0.0f;
#pragma unroll
            for (int u = 0; u < U; ++u) acc += float(ed[u].count) * v[u];
        }
    }
    __syncwarp();
#pragma unroll
    for (int k = 1; k < L; k <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
    const facetcu_surface_optics& o = r.optics;
    const float h = (r.denom == 0u ? sky : (float(r.skyc) * sky + acc) / float(r.denom)) +
                    o.direct_irradiance;
    const float other = __shfl_xor_sync(0xffffffffu, h, L);  // the facet's other side
    if (!valid || eg != 0) return 0.0f;
    const float t = o.emission + o.reflectance * h + o.transmittance * other;
    // GLSL mix(x, y, a) = x * (1 - a) + y * a
    const float b = old * (1.0f - relax) + t * relax;
    Bout[s] = b;
    return fabsf(b - old);
}
__device__ __forceinline__ void publish_delta(float delta, uint32_t* max_delta_bits)
{
    __shared__ float block_delta[8];
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) delta = fmaxf(delta, __shfl_xor_sync(0xffffffffu, delta, k));
    if ((threadIdx.x & 31) == 0) block_delta[threadIdx.x >> 5] = delta;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) delta = fmaxf(delta, block_delta[w]);
        atomicMax(max_delta_bits, __float_as_uint(delta));
    }
}

template <int L, bool kEarly>
__global__ void __launch_bounds__(256) k_jacobi_rows(
    uint32_t facets, const uint32_t* __restrict__ rows, const facetcu_csr_edge* __restrict__ edges,
    const uint32_t* __restrict__ denom, const uint32_t* __restrict__ skyc,
    const facetcu_surface_optics* __restrict__ optics, float sky, float relax,
    const float* Bin, float* Bout, uint32_t* max_delta_bits)
{
    if (kEarly) start_next();
    const uint32_t s = side_of(blockIdx.x, threadIdx.x, L);
    const bool valid = (s >> 1) < facets;
    const SideRow r = load_row<L>(valid, s, rows, denom, skyc, optics);
    if (kEarly) wait_for_previous();
    publish_delta(sweep_row<L>(valid, s, r, edges, sky, relax, Bin, Bout), max_delta_bits);
}

// Lanes of a side for rows of `mean` edges.  A sweep in us (k_jacobi_any; rows of
// half to one and a half times the mean) with 1, 4, 8 and 16 lanes, and with one
// thread per facet:
//     mean              2     4     8    12    20    32    48    64
//     40,000 sides 1  4.4   5.3   6.4   8.4  10.5  14.6  18.7  24.7
//                  4  4.3   6.3   6.4   6.4   8.4   8.5  10.5  12.5
//                  8  6.3   6.3   6.4   6.4   8.4   8.5  10.5  12.5
//                 16  8.4   8.4   8.4   8.4   8.4   9.0  10.4  11.7
//             thread  6.4   7.4   8.4  10.5  10.9  14.5  18.5  20.9
//     1,000,000    1   12    19    35    58   107   180   271
//                  4   27    27    37    53    76   121   182
//                  8   49    50    52    59    77   108   155
//                 16   95    96    97    99   103   115   157
//             thread   23    31    46    68   101   162   230
// (Short rows of large graphs leave most of many lanes idle; below 2,048 sides all
// but 1 take the 4.3 us of a launch up to 20 edges.)
constexpr __host__ __device__ int lanes_for(uint64_t mean)
{
    return mean < 4 ? 1 : mean < 10 ? 4 : mean < 48 ? 8 : 16;
}

// The sweep where only the device knows the number of edges, rows[surfaces]: a
// grid of resident blocks walks the sides, with lanes by the same rule.  (With the
// lanes of the longest rows whatever the graph, a million sides of 1 to 8 edges
// took 92 to 107 us a sweep; one thread per facet 19 to 46, this 10 to 37.)
template <int L>
__device__ __forceinline__ float sweep_rows_of(uint32_t surfaces, const uint32_t* __restrict__ rows,
                                               const facetcu_csr_edge* __restrict__ edges,
                                               const uint32_t* __restrict__ denom,
                                               const uint32_t* __restrict__ skyc,
                                               const facetcu_surface_optics* __restrict__ optics,
                                               float sky, float relax, const float* Bin, float* Bout)
{
    float delta = 0.0f;
    const uint32_t blocks = (surfaces + 256u / L - 1u) / (256u / L);
    for (uint32_t b = blockIdx.x; b < blocks; b += gridDim.x) {
        const uint32_t s = side_of(b, threadIdx.x, L);
        const bool valid = s < surfaces;
        const SideRow r = load_row<L>(valid, s, rows, denom, skyc, optics);
        delta = fmaxf(delta, sweep_row<L>(valid, s, r, edges, sky, relax, Bin, Bout));
    }
    return delta;
}
__global__ void __launch_bounds__(256) k_jacobi_any(
    uint32_t surfaces, const uint32_t* __restrict__ rows, const facetcu_csr_edge* __restrict__ edges,
    const uint32_t* __restrict__ denom, const uint32_t* __restrict__ skyc,
    const facetcu_surface_optics* __restrict__ optics, float sky, float relax, const float* Bin,
    float* Bout, uint32_t* max_delta_bits)
{
    const int lanes = lanes_for(rows[surfaces] / surfaces);
    auto sweep = [&](auto L) {
        return sweep_rows_of<decltype(L)::value>(surfaces, rows, edges, denom, skyc, optics, sky, relax,
                                                 Bin, Bout);
    };
    float delta;
    if (lanes == 1) delta = sweep(std::integral_constant<int, 1>{});
    else if (lanes == 4) delta = sweep(std::integral_constant<int, 4>{});
    else if (lanes == 8) delta = sweep(std::integral_constant<int, 8>{});
    else delta = sweep(std::integral_constant<int, 16>{});
    publish_delta(delta, max_delta_bits);
}

// ---- all sweeps of a small graph in one launch ----------------------------
// A sweep of the smallest graphs is shorter than a launch, even one that begins
// early.  Here a cluster of 16 blocks runs all of them: every block holds the
// whole radiosity twice (this sweep's and the next), its share of the sides and
// their edges in shared memory, and writes its new values into the others'.
// Bound by that exchange and the cluster's barrier: 1 us a sweep for 1,152
// sides, 2.5 for 8,192 (with blocks that wait on a count of received bytes
// instead, 2.2 by bulk copies and 3.2 by asynchronous stores).  A call of 64 sweeps
// in us, in early launches / here:
//     edges     7,000      16,000     33,000     50,000     70,000     100,000
//       256   157 / 131  158 / 159  196 / 281  248 / 283  255 / 359  337 / 465
//       768   161 / 122  159 / 127  176 / 148  195 / 172  189 / 196  229 / 233
//     1,152   169 / 125  170 / 138  171 / 147  191 / 162  182 / 176  205 / 200
//     2,048   180 / 129  175 / 133  181 / 153  181 / 153  223 / 165  200 / 203
//     3,200   190 / 145  180 / 148  187 / 158  199 / 159  199 / 170  216 / 182
//     4,096              195 / 150  188 / 162  202 / 162  213 / 173  218 / 191
// so rows of more than 64 edges, which two lanes read alone, go to the launches.
// (8,192 sides of 98,058 edges: 243 / 249.  Four lanes a side: 125 for the first and
// 279 for the last; eight blocks: 304 for the last.)  Setting up costs some
// launches: 12 sweeps take 59 us and 57 on 256 sides, 65 and 67 on 1,152.
constexpr uint32_t kCtas = 16, kClusterThreads = 1024, kGroup = 16, kDeltas = 64;
constexpr int kClusterLanes = 2;
constexpr uint32_t kClusterSides = 4096, kClusterSweeps = 12;
constexpr uint64_t kClusterEdges = 100000, kClusterMean = 64;
constexpr size_t kClusterShared = 227 * 1024 - 1024;  // (static arrays besides)

struct ClusterShape {
    uint32_t padded;  // sides, the same whole number of groups for every block
    uint32_t owned;   // a block's, whole groups
    uint32_t words;   // edges that fit; the rest is read from memory
};

// Sides go to the blocks in groups of 16 in turn, so that rows of different
// lengths even out.
__device__ __forceinline__ uint32_t owned_side(uint32_t j, uint32_t rank)
{
    return (rank + kCtas * (j / kGroup)) * kGroup + j % kGroup;
}

template <int L>
__global__ void __launch_bounds__(kClusterThreads, 1) k_jacobi_cluster(
    ClusterShape shape, uint32_t surfaces, const uint32_t* __restrict__ rows,
    const facetcu_csr_edge* __restrict__ edges, const uint32_t* __restrict__ denom,
    const uint32_t* __restrict__ skyc, const facetcu_surface_optics* __restrict__ optics, float sky,
    float relax, const float* first, float* out_even, float* out_odd, uint32_t sweeps,
    uint32_t* max_delta_bits)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), tid = threadIdx.x, lane = tid & 31u;
    extern __shared__ float4 shared4[];
    float* x = reinterpret_cast<float*>(shared4);                       // [2][padded]
    float4* opt = shared4 + 2 * shape.padded / 4;                       // [owned]
    float2* norm = reinterpret_cast<float2*>(opt + shape.owned);        // [owned]
    uint32_t* start = reinterpret_cast<uint32_t*>(norm + shape.owned);  // [owned + 4]
    uint32_t* words = start + shape.owned + 4;
    __shared__ uint32_t warp_sum[kClusterThreads / 32];
    __shared__ uint32_t block_delta[kDeltas];  // of kDeltas sweeps, sent off together
    if (tid < kDeltas) block_delta[tid] = 0;
    for (uint32_t i = tid; i < shape.padded; i += kClusterThreads) x[i] = i < surfaces ? first[i] : 0.0f;
    uint32_t base = 0;
    for (uint32_t j0 = 0; j0 < shape.owned; j0 += kClusterThreads) {
        const uint32_t j = j0 + tid, s = owned_side(j, rank);
        const bool on = j < shape.owned && s < surfaces;
        const uint32_t n = on ? rows[s + 1] - rows[s] : 0u;
        uint32_t incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        if (lane == 31u) warp_sum[tid >> 5] = incl;
        __syncthreads();
        uint32_t before = base, all = 0;
        for (uint32_t w = 0; w < kClusterThreads / 32; ++w) {
            if (w < tid >> 5) before += warp_sum[w];
            all += warp_sum[w];
        }
        if (j < shape.owned) {
            start[j] = before + incl - n;
            if (j + 1 == shape.owned) start[j + 1] = before + incl;
            opt[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            norm[j] = make_float2(0.0f, 0.0f);
            if (on) {
                const facetcu_surface_optics o = optics[s];
                opt[j] = make_float4(o.reflectance, o.transmittance, o.emission, o.direct_irradiance);
                norm[j] = make_float2(float(skyc[s]), float(denom[s]));
            }
        }
        base += all;
        __syncthreads();
    }
    for (uint32_t j = tid / 8; j < shape.owned; j += kClusterThreads / 8) {
        const uint32_t s = owned_side(j, rank);
        if (s >= surfaces) continue;
        const uint32_t from = rows[s], n = rows[s + 1] - from, at = start[j];
        for (uint32_t e = tid % 8; e < n && at + e < shape.words; e += 8) {
            const facetcu_csr_edge ed = edges[from + e];
            words[at + e] = ed.neighbor << 16 | ed.count;
        }
    }
    cluster.sync();
    constexpr int U = 2;
    for (uint32_t it = 0; it < sweeps; ++it) {
        const float* now = x + (it & 1u ? shape.padded : 0u);
        float* next = x + (it & 1u ? 0u : shape.padded);
        float delta = 0.0f;
        for (uint32_t j = tid / L; j < shape.owned; j += kClusterThreads / L) {
            const uint32_t at = start[j], n = start[j + 1] - at, s = owned_side(j, rank);
            const uint32_t held = at >= shape.words ? 0u : min(n, shape.words - at);
            float acc = 0.0f;
            uint32_t e = tid % L;
            for (; e < held; e += L * U) {
                uint32_t w[U];
                float v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) w[u] = e + u * L < held ? words[at + e + u * L] : 0u;
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = now[w[u] >> 16];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (e + u * L < held) acc += float(w[u] & 0xffffu) * v[u];
            }
            e = held + (tid % L + L - held % L) % L;
            if (e < n) {
                const uint32_t from = rows[s];
                for (; e < n; e += L) {
                    const facetcu_csr_edge ed = edges[from + e];
                    acc += float(ed.count) * now[ed.neighbor];
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = 1; k < L; k <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
            const float4 o = opt[j];
            const float2 d = norm[j];
            const float h = (d.y == 0.0f ? sky : (d.x * sky + acc) / d.y) + o.w;
            const float other = __shfl_xor_sync(0xffffffffu, h, L);  // the facet's other side
            if (tid % L == 0) {
                const float old = now[s], t = o.z + o.x * h + o.y * other;
                const float b = s < surfaces ? old * (1.0f - relax) + t * relax : 0.0f;
                next[s] = b;
                delta = fmaxf(delta, fabsf(b - old));
            }
        }
        const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(delta));
        if (lane == 0) atomicMax(&block_delta[it % kDeltas], most);
        __syncthreads();
        // this block's values to the others, two warps to each, 16 bytes a lane
        for (uint32_t w = tid >> 5; w < 2 * (kCtas - 1); w += kClusterThreads / 32) {
            float* there = cluster.map_shared_rank(next, (rank + 1 + w / 2) % kCtas);
            for (uint32_t p = (w & 1u) * 32 + lane; p < shape.owned / 4; p += 64) {
                const uint32_t s = owned_side(4 * p, rank);
                *reinterpret_cast<float4*>(there + s) = *reinterpret_cast<const float4*>(next + s);
            }
        }
        if (it % kDeltas == kDeltas - 1 || it + 1 == sweeps) {
            // (a global atomic in every sweep would have to be waited for at the barrier)
            const uint32_t k = it - it % kDeltas + tid;
            if (k <= it && tid < kDeltas) {
                atomicMax(max_delta_bits + k, block_delta[tid]);
                block_delta[tid] = 0;
            }
        }
        cluster.sync();
    }
    for (uint32_t j = tid; j < shape.owned; j += kClusterThreads) {
        const uint32_t s = owned_side(j, rank);
        if (s >= surfaces) continue;
        out_even[s] = x[s];
        out_odd[s] = x[shape.padded + s];
    }
}

// FacetrtVulkan::incidentIrradiance / incidentIrradianceCpu
// (facetrt_vulkan.cpp:1360-1399, facetrtcore.cpp:1531-1559): FP64 gather.
__global__ void __launch_bounds__(128) k_incident(
    uint32_t surfaces, const uint32_t* rows, const facetcu_csr_edge* edges, const uint32_t* denom,
    const uint32_t* skyc, const facetcu_surface_optics* optics, float sky, const float* B,
    float* out)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= surfaces) return;
    double diffuse = sky;
    const uint32_t d = denom[s];
    if (d != 0u) {
        diffuse = double(skyc[s]) * double(sky);
        for (uint32_t e = rows[s]; e < rows[s + 1]; ++e) {
            const facetcu_csr_edge ed = edges[e];
            diffuse += double(ed.count) * double(B[ed.neighbor]);
        }
        diffuse /= double(d);
    }
    out[s] = fmaxf(0.0f, float(diffuse) + optics[s].direct_irradiance);
}

}  // namespace

namespace {

template <bool kEarly>
void sweep_rows(const DeviceGraph& g, const facetcu_surface_optics* d_optics, float sky,
                float relaxation, const float* d_in, float* d_out, uint32_t* d_max_delta_bits,
                cudaStream_t s)
{
    const uint32_t facets = g.surfaces / 2u;
    if (!facets) return;
    auto launch = [&](auto lanes) {
        constexpr int L = decltype(lanes)::value;
        const unsigned grid = unsigned((uint64_t(g.surfaces) * L + 255) / 256);
        const uint32_t *rows = g.row_offsets.as<uint32_t>(), *denom = g.denominators.as<uint32_t>(),
                       *skyc = g.sky.as<uint32_t>();
        const facetcu_csr_edge* edges = g.edges.as<facetcu_csr_edge>();
        if (kEarly)
            launch_early(k_jacobi_rows<L, true>, grid, 256, 0, s, facets, rows, edges, denom, skyc,
                         d_optics, sky, relaxation, d_in, d_out, d_max_delta_bits);
        else
            k_jacobi_rows<L, false><<<grid, 256, 0, s>>>(facets, rows, edges, denom, skyc, d_optics,
                                                         sky, relaxation, d_in, d_out,
                                                         d_max_delta_bits);
    };
    switch (lanes_for(g.nnz / g.surfaces)) {
    case 1: launch(std::integral_constant<int, 1>{}); break;
    case 4: launch(std::integral_constant<int, 4>{}); break;
    case 8: launch(std::integral_constant<int, 8>{}); break;
    default: launch(std::integral_constant<int, 16>{}); break;
    }
    FCU_LAUNCH("k_jacobi_rows");
}

}  // namespace

// (The caller's arrays may have been written by the kernel just before: no
// early start here.)
void jacobi_sweep_raw(uint32_t surfaces, const uint32_t* rows, const facetcu_csr_edge* edges,
                      const uint32_t* denom, const uint32_t* skyc,
                      const facetcu_surface_optics* d_optics, float sky, float relaxation,
                      const float* d_in, float* d_out, uint32_t* d_max_delta_bits, cudaStream_t s)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned most = unsigned((uint64_t(surfaces) * 16 + 255) / 256);
    k_jacobi_any<<<std::min(most, 8u * unsigned(std::max(sms, 1))), 256, 0, s>>>(
        surfaces, rows, edges, denom, skyc, d_optics, sky, relaxation, d_in, d_out, d_max_delta_bits);
    FCU_LAUNCH("k_jacobi_any");
}

void jacobi_sweep(const DeviceGraph& g, bool planned, const facetcu_surface_optics* d_optics,
                  float sky, float relaxation, const float* d_in, float* d_out, uint32_t* d_max_delta_bits,
                  bool follows, cudaStream_t s)
{
    if (planned) {
        column_jacobi(g, d_optics, sky, relaxation, d_in, d_out, d_max_delta_bits, s);
        return;
    }
    (follows ? sweep_rows<true> : sweep_rows<false>)(g, d_optics, sky, relaxation, d_in, d_out,
                                                     d_max_delta_bits, s);
}

bool jacobi_sweeps_cluster(const DeviceGraph& g, const facetcu_surface_optics* d_optics, float sky,
                           float relaxation, float* d_in, float* d_other, uint32_t sweeps,
                           uint32_t* d_max_delta_bits, cudaStream_t s)
{
    const uint32_t S = g.surfaces;
    if (sweeps < kClusterSweeps || S < 2 || S > kClusterSides || g.nnz > kClusterEdges ||
        g.nnz > kClusterMean * S || g.max_count > 0xffffu)
        return false;
    ClusterShape shape;
    const uint32_t groups = (S + kGroup - 1) / kGroup;
    shape.owned = (groups + kCtas - 1) / kCtas * kGroup;
    shape.padded = shape.owned * kCtas;
    const size_t fixed = size_t(shape.padded) * 8 + size_t(shape.owned) * 28 + 16;
    // a block whose share of the edges is larger than what it has room for
    // reads the rest from memory
    const size_t room = (kClusterShared - fixed) / 4;
    shape.words = uint32_t(std::min<size_t>(room, g.nnz / kCtas * 2 + 1024));
    auto kernel = k_jacobi_cluster<kClusterLanes>;
    const size_t shared = fixed + size_t(shape.words) * 4;
    // (the limits belong to the function, not to this context: always the most)
    FCU_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(kClusterShared)));
    FCU_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t config{};
    config.gridDim = kCtas;
    config.blockDim = kClusterThreads;
    config.dynamicSmemBytes = shared;
    config.stream = s;
    cudaLaunchAttribute cluster{};
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim = {kCtas, 1, 1};
    config.attrs = &cluster;
    config.numAttrs = 1;
    int fits = 0;
    if (cudaOccupancyMaxActiveClusters(&fits, kernel, &config) != cudaSuccess || fits < 1) {
        cudaGetLastError();
        return false;
    }
    // after `sweeps` sweeps the values lie where single sweeps would leave them
    FCU_CHECK(cudaLaunchKernelEx(&config, kernel, shape, S, (const uint32_t*)g.row_offsets.ptr,
                                 (const facetcu_csr_edge*)g.edges.ptr,
                                 (const uint32_t*)g.denominators.ptr, (const uint32_t*)g.sky.ptr,
                                 d_optics, sky, relaxation, (const float*)d_in, d_in, d_other, sweeps,
                                 d_max_delta_bits));
    return true;
}

void incident_irradiance(const DeviceGraph& g, const facetcu_surface_optics* d_optics, float sky,
                         const float* d_radiosity, float* d_out, cudaStream_t s)
{
    if (!g.surfaces) return;
    k_incident<<<(g.surfaces + 127) / 128, 128, 0, s>>>(
        g.surfaces, g.row_offsets.as<uint32_t>(), g.edges.as<facetcu_csr_edge>(),
        g.denominators.as<uint32_t>(), g.sky.as<uint32_t>(), d_optics, sky, d_radiosity, d_out);
    FCU_LAUNCH("k_incident");
}

}  // namespace facetcu
