// solve.cu — the reference's single-RHS Jacobi sweep and incident irradiance.
//
// k_jacobi_rows is the sweep of the reference's radiosity.comp:49-106
// (FacetrtVulkan::solve): FP32 gather over the count-form CSR, both sides of a
// facet updated together, mix() relaxation, max|dB| as an atomicMax over float
// bits.  It serves the graphs that column.cu's plan is not made for (few
// edges, short rows) and callers that bring their own arrays.
#include "internal.h"

namespace facetcu {
namespace {

// L lanes per side, so a facet's two rows are read at once by 2 L lanes:
// each lane has U edges in flight and the chain of dependent loads of a row
// (offsets, edge words, neighbour values) is paid once for all of them.
// (One thread per facet walked ~30 such chains: 7.2 us per sweep on the
// 4,096-facet scene of 98,000 edges, 4.1 here.)  L follows the mean row length.
template <int L>
__global__ void __launch_bounds__(256) k_jacobi_rows(
    uint32_t facets, const uint32_t* __restrict__ rows, const facetcu_csr_edge* __restrict__ edges,
    const uint32_t* __restrict__ denom, const uint32_t* __restrict__ skyc,
    const facetcu_surface_optics* __restrict__ optics, float sky, float relax,
    const float* __restrict__ Bin, float* __restrict__ Bout, uint32_t* max_delta_bits)
{
    constexpr int U = 4;
    __shared__ float block_delta[8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t eg = lane % L;
    const uint32_t s = (blockIdx.x * 256 + threadIdx.x) / L;  // side
    float delta = 0.0f;
    // whole warps stay for the shuffles
    const bool valid = (s >> 1) < facets;
    float acc = 0.0f, old = 0.0f;
    uint32_t d = 0, sc = 0;
    facetcu_surface_optics o{};
    if (valid) {
        const uint32_t start = rows[s], end = rows[s + 1];
        d = denom[s];
        if (eg == 0) {
            sc = skyc[s];
            o = optics[s];
            old = Bin[s];
        }
        for (uint32_t e = start + eg; e < end; e += L * U) {
            facetcu_csr_edge ed[U];
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ed[u] = {0u, 0u};
                if (e + u * L < end) ed[u] = edges[e + u * L];
            }
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = e + u * L < end ? Bin[ed[u].neighbor] : 0.0f;
#pragma unroll
            for (int u = 0; u < U; ++u) acc += float(ed[u].count) * v[u];
        }
    }
#pragma unroll
    for (int k = 1; k < L; k <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
    const float h = (d == 0u ? sky : (float(sc) * sky + acc) / float(d)) + o.direct_irradiance;
    const float other = __shfl_xor_sync(0xffffffffu, h, L);  // the facet's other side
    if (valid && eg == 0) {
        const float t = o.emission + o.reflectance * h + o.transmittance * other;
        // GLSL mix(x, y, a) = x * (1 - a) + y * a
        const float b = old * (1.0f - relax) + t * relax;
        Bout[s] = b;
        delta = fabsf(b - old);
    }
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) delta = fmaxf(delta, __shfl_xor_sync(0xffffffffu, delta, k));
    if (lane == 0) block_delta[warp] = delta;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) delta = fmaxf(delta, block_delta[w]);
        atomicMax(max_delta_bits, __float_as_uint(delta));
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

void jacobi_sweep_raw(uint32_t surfaces, uint64_t edges_hint, const uint32_t* rows,
                      const facetcu_csr_edge* edges, const uint32_t* denom, const uint32_t* skyc,
                      const facetcu_surface_optics* d_optics, float sky, float relaxation,
                      const float* d_in, float* d_out, uint32_t* d_max_delta_bits, cudaStream_t s)
{
    const uint32_t facets = surfaces / 2u;
    if (!facets) return;
    auto launch = [&](auto kernel, uint32_t lanes) {
        const uint64_t threads = uint64_t(surfaces) * lanes;
        kernel<<<unsigned((threads + 255) / 256), 256, 0, s>>>(facets, rows, edges, denom, skyc,
                                                              d_optics, sky, relaxation, d_in,
                                                              d_out, d_max_delta_bits);
    };
    const uint64_t mean = edges_hint / surfaces;
    if (mean < 8) launch(k_jacobi_rows<4>, 4);
    else if (mean < 48) launch(k_jacobi_rows<8>, 8);
    else launch(k_jacobi_rows<16>, 16);
    FCU_LAUNCH("k_jacobi_rows");
}

void jacobi_sweep(const DeviceGraph& g, const facetcu_surface_optics* d_optics, float sky,
                  float relaxation, const float* d_in, float* d_out, uint32_t* d_max_delta_bits,
                  cudaStream_t s)
{
    if (g.column.state == ColumnPlan::kMade) {
        column_jacobi(g, d_optics, sky, relaxation, d_in, d_out, d_max_delta_bits, s);
        return;
    }
    jacobi_sweep_raw(g.surfaces, g.nnz, g.row_offsets.as<uint32_t>(), g.edges.as<facetcu_csr_edge>(),
                     g.denominators.as<uint32_t>(), g.sky.as<uint32_t>(), d_optics, sky, relaxation,
                     d_in, d_out, d_max_delta_bits, s);
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
