// geometry.cu — the checks of setGeometry on the device.
//
// FacetrtVulkan::validateGeometry (facetrt_vulkan.cpp:425-453) refuses the
// first vertex whose position is not finite or whose normal is not of unit
// length, and the bounds of the positions frame the raster.  On the host the
// pass over the vertices took 3 ms for 200,000 facets, more than the raster
// build that follows; here it is one read of the uploaded vertices (compiled
// with -fmad=false: the normal's length rounds as the host's did).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "internal.h"

namespace facetcu {
namespace {

struct Result {
    uint32_t bad_position, bad_normal;
    uint32_t lo[3], hi[3];  // ordered keys
};
static_assert(sizeof(Result) == 32, "five minima, three maxima");

// Order-preserving key of a finite float.
__device__ __host__ inline uint32_t key_of(uint32_t bits)
{
    return bits & 0x80000000u ? ~bits : bits | 0x80000000u;
}
inline float value_of(uint32_t key)
{
    const uint32_t bits = key & 0x80000000u ? key & 0x7fffffffu : ~key;
    float f;
    std::memcpy(&f, &bits, 4);
    return f;
}

__global__ void __launch_bounds__(256) k_check_geometry(const float* __restrict__ v, uint64_t count,
                                                        Result* r)
{
    // Warps meet in shared memory first: with six atomics a warp on the one
    // sector of *r those took 40 us of the 146 that setGeometry takes for 600,000
    // vertices; 111 so.
    __shared__ Result block;
    if (threadIdx.x < 8)
        reinterpret_cast<uint32_t*>(&block)[threadIdx.x] = threadIdx.x < 5 ? 0xffffffffu : 0u;
    __syncthreads();
    uint32_t bad_position = 0xffffffffu, bad_normal = 0xffffffffu;
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride) {
        const float2* q = reinterpret_cast<const float2*>(v + 6 * i);
        const float2 a = q[0], b = q[1], c = q[2];
        const float p[3] = {a.x, a.y, b.x}, n[3] = {b.y, c.x, c.y};
        bool finite = true;
        for (int k = 0; k < 3; ++k) {
            finite &= isfinite(p[k]);
            lo[k] = fminf(lo[k], p[k]);
            hi[k] = fmaxf(hi[k], p[k]);
        }
        if (!finite) bad_position = min(bad_position, uint32_t(i));
        const float len = sqrtf(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        if (!(len > 0.99f && len < 1.01f)) bad_normal = min(bad_normal, uint32_t(i));
    }
    const bool first = (threadIdx.x & 31) == 0;
    bad_position = __reduce_min_sync(0xffffffffu, bad_position);
    bad_normal = __reduce_min_sync(0xffffffffu, bad_normal);
    if (first) {
        atomicMin(&block.bad_position, bad_position);
        atomicMin(&block.bad_normal, bad_normal);
    }
    for (int k = 0; k < 3; ++k) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, key_of(__float_as_uint(lo[k])));
        const uint32_t h = __reduce_max_sync(0xffffffffu, key_of(__float_as_uint(hi[k])));
        if (first) {
            atomicMin(&block.lo[k], l);
            atomicMax(&block.hi[k], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        const uint32_t x = reinterpret_cast<const uint32_t*>(&block)[threadIdx.x];
        uint32_t* out = reinterpret_cast<uint32_t*>(r) + threadIdx.x;
        if (threadIdx.x < 5) atomicMin(out, x);
        else atomicMax(out, x);
    }
}

// The same check on the host.
GeometryCheck check_on_host(const facetcu_vertex* v, uint64_t count)
{
    GeometryCheck r{~0u, ~0u, {FLT_MAX, FLT_MAX, FLT_MAX}, {-FLT_MAX, -FLT_MAX, -FLT_MAX}};
    for (uint64_t i = 0; i < count; ++i) {
        bool finite = true;
        for (int k = 0; k < 3; ++k) {
            const float p = v[i].position[k];
            finite = finite && std::isfinite(p);
            r.lo[k] = std::min(r.lo[k], p);
            r.hi[k] = std::max(r.hi[k], p);
        }
        const float* n = v[i].normal;
        const float len = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        if (!finite) r.bad_position = std::min(r.bad_position, uint32_t(i));
        if (!(len > 0.99f && len < 1.01f)) r.bad_normal = std::min(r.bad_normal, uint32_t(i));
    }
    return r;
}

// Vertices up to which the host is faster than a kernel and its answer's way back:
// setGeometry of 12 facets 10 us against 20, of 500 18 against 24, of 1,000 26
// against 29, of 5,000 80 against 31 (about 5 ns a vertex).
constexpr uint64_t kHostVertices = 3600;

}  // namespace

bool check_small_geometry(const facetcu_vertex* vertices, uint64_t count, GeometryCheck& check)
{
    if (count > kHostVertices) return false;
    check = check_on_host(vertices, count);
    return true;
}

GeometryCheck check_geometry(const facetcu_vertex* d_vertices, uint64_t count, Workspace& ws,
                             cudaStream_t s)
{
    ScratchBuffer buf(ws);
    Result* d = static_cast<Result*>(buf.reserve(sizeof(Result)));
    Result r;
    std::memset(&r, 0xff, sizeof(r));
    for (uint32_t& h : r.hi) h = 0;
    FCU_CHECK(cudaMemcpyAsync(d, &r, sizeof(r), cudaMemcpyHostToDevice, s));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned grid = unsigned(std::min<uint64_t>((count + 255) / 256, uint64_t(std::max(sms, 1)) * 8));
    k_check_geometry<<<grid, 256, 0, s>>>(reinterpret_cast<const float*>(d_vertices), count, d);
    FCU_LAUNCH("k_check_geometry");
    FCU_CHECK(cudaMemcpyAsync(&r, d, sizeof(r), cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaStreamSynchronize(s));
    GeometryCheck c;
    c.bad_position = r.bad_position;
    c.bad_normal = r.bad_normal;
    for (int k = 0; k < 3; ++k) {
        c.lo[k] = value_of(r.lo[k]);
        c.hi[k] = value_of(r.hi[k]);
    }
    return c;
}

GeometryCheck check_geometry_in_pieces(const facetcu_vertex* vertices, uint64_t count,
                                       Workspace& ws, cudaStream_t s)
{
    constexpr uint64_t kPiece = 1u << 17;  // 3 MB
    ScratchBuffer buf(ws);
    facetcu_vertex* d = static_cast<facetcu_vertex*>(
        buf.reserve(std::min(count, kPiece) * sizeof(facetcu_vertex)));
    GeometryCheck all{0xffffffffu, 0xffffffffu, {FLT_MAX, FLT_MAX, FLT_MAX}, {-FLT_MAX, -FLT_MAX, -FLT_MAX}};
    for (uint64_t first = 0; first < count; first += kPiece) {
        const uint64_t n = std::min(kPiece, count - first);
        FCU_CHECK(cudaMemcpyAsync(d, vertices + first, n * sizeof(facetcu_vertex),
                                  cudaMemcpyHostToDevice, s));
        const GeometryCheck c = check_geometry(d, n, ws, s);
        if (c.bad_position != 0xffffffffu)
            all.bad_position = std::min(all.bad_position, uint32_t(first) + c.bad_position);
        if (c.bad_normal != 0xffffffffu)
            all.bad_normal = std::min(all.bad_normal, uint32_t(first) + c.bad_normal);
        for (int a = 0; a < 3; ++a) {
            all.lo[a] = std::min(all.lo[a], c.lo[a]);
            all.hi[a] = std::max(all.hi[a], c.hi[a]);
        }
    }
    return all;
}

}  // namespace facetcu
