// raster.cu — global-line visibility: orthographic A-buffer raster of every
// facet along each direction, per-pixel depth chains, pair emission.
//
// Semantics are those of the reference's CPU backend (CpuRasterizer,
// buildCpuGraph, computeCpuSunlit: facetrtcore.cpp:1212-1474) so that the
// integer counts are identical:
//   * the projection, edge functions and interpolated depth use the same
//     float expressions in the same order; this file is compiled with
//     -fmad=false so no multiply-add is fused, as in the reference build;
//   * coverage is the inclusive edge test at pixel centres (:1315-1318);
//   * fragments of a pixel are ordered as std::sort (GCC's introsort)
//     orders them when given the reference's append order (tile-major,
//     then facet index): chains of <= 16 are stably sorted by depth, longer
//     chains replay the introsort step for step.
//
// GB300 layout: instead of a fixed W x H x L A-buffer (512 MB per direction
// at 1024^2 x 64) every pixel heads a list of its fragments, in one pool for a
// whole chunk of directions, so a single launch covers all 40 directions, each
// triangle is rasterised once, and HBM holds only real fragments.  A block
// takes its room in the pool with one atomic.  A pool that turns out too small
// is grown to the exact number and the chunk rasterised again.  A facet's
// fragments are counted by the threads that rasterise it, not fragment by
// fragment when the lists are resolved.  The sun pass needs a pixel's nearest
// fragment and their number only: no lists, two atomics a fragment.
#include <algorithm>

#include "internal.h"

namespace facetcu {
namespace {

// Who takes a triangle, by the area of its bounding box.  Build of the graph,
// us, 4,096 facets of terrain (boxes of some 500 pixels) / 200,000 facets of
// forest (most below 10, the ground's about 100), 40 directions of 1024^2:
//   a thread up to 8, 16, 32 pixels:  925 / 5288,  929 / 2095,  876 / 2005
//   above, 4, 8, 16, 32 lanes:        839 / 1709,  848 / 1777,  870 / 1904,
//                                     894 / 2194
// and the one direction of the sun pass, when it had lists too, with 4, 8, 32
// lanes: 144 / 157, 121 / 155, 110 / 169.
constexpr uint32_t kSmallPixels = 32;  // (a thread's covered pixels are bits of a word)
constexpr uint32_t kMidLanes = 8;
constexpr uint32_t kBigPixels = 1024;  // above: blocks
constexpr int kFast = 8;               // chains ordered in registers
constexpr uint32_t kMidChain = 64;     // per-thread chain capacity of the middle resolve
constexpr uint32_t kDeepChain = 1024;  // capacity of the deep-chain resolve
constexpr uint32_t kResolvePixels = 2048;  // pixels of a resolving block
constexpr uint32_t kKeyMask = 0x7fffffffu;

// What a raster kernel looks at, by value in its parameters: __constant__
// copies would be one per device, and another context's build on its own stream
// would change them between this one's kernels.
constexpr uint32_t kMaxViews = 64;
struct Scene {
    RasterFrame frame;
    RasterView views[kMaxViews];
};

struct Projected {
    float x[3], y[3], d[3];
};

__device__ __forceinline__ float dot3(const float a[3], float b0, float b1, float b2)
{
    return a[0] * b0 + a[1] * b1 + a[2] * b2;
}

// facetrtcore.cpp:1259-1275
__device__ __forceinline__ void project_vertex(const RasterFrame& frame, float px, float py,
                                               float pz, uint32_t tile, const RasterView& v,
                                               float& x, float& y, float& d)
{
    const float r = frame.radius;
    const float rx = (px + frame.tile_dx[tile]) - frame.center[0];
    const float ry = py - frame.center[1];
    const float rz = (pz + frame.tile_dz[tile]) - frame.center[2];
    x = (0.5f + 0.5f * dot3(v.right, rx, ry, rz) / r) * float(frame.width);
    y = (0.5f + 0.5f * dot3(v.up, rx, ry, rz) / r) * float(frame.height);
    d = 0.5f - dot3(v.view, rx, ry, rz) / (2.0f * r);
}

// The triangles as three planes of 16 bytes a facet (corners, then the first
// corner's normal): a warp of facets reads them in 12 wavefronts, where the
// vertices' 24-byte records take some 200 and bounded the raster of 200,000
// facets.
__global__ void k_planes(const facetcu_vertex* __restrict__ V, uint32_t facets,
                         float4* __restrict__ planes)
{
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= facets) return;
    const facetcu_vertex &a = V[3 * f], &b = V[3 * f + 1], &c = V[3 * f + 2];
    planes[f] = make_float4(a.position[0], a.position[1], a.position[2], b.position[0]);
    planes[facets + f] = make_float4(b.position[1], b.position[2], c.position[0], c.position[1]);
    planes[2 * size_t(facets) + f] =
        make_float4(c.position[2], a.normal[0], a.normal[1], a.normal[2]);
}

struct Facet {
    float4 q0, q1, q2;
};
__device__ __forceinline__ Facet load_facet(const RasterFrame& frame, const float4* planes, uint32_t f)
{
    const size_t F = frame.facets;
    return {__ldg(planes + f), __ldg(planes + F + f), __ldg(planes + 2 * F + f)};
}
__device__ __forceinline__ uint32_t facing(const Facet& t, const RasterView& v)
{
    return dot3(v.view, t.q2.y, t.q2.z, t.q2.w) >= 0.0f ? 0u : 1u;
}
__device__ __forceinline__ void project(const RasterFrame& frame, const Facet& t, uint32_t tile,
                                        const RasterView& v, Projected& p)
{
    project_vertex(frame, t.q0.x, t.q0.y, t.q0.z, tile, v, p.x[0], p.y[0], p.d[0]);
    project_vertex(frame, t.q0.w, t.q1.x, t.q1.y, tile, v, p.x[1], p.y[1], p.d[1]);
    project_vertex(frame, t.q1.z, t.q1.w, t.q2.x, tile, v, p.x[2], p.y[2], p.d[2]);
}
// The same by kLanes lanes: they take a corner each and exchange.
template <uint32_t kLanes>
__device__ __forceinline__ void project_lanes(const RasterFrame& frame, const Facet& t, uint32_t tile,
                                              const RasterView& v, Projected& p)
{
    const uint32_t c = (threadIdx.x % kLanes) % 3u;
    const float px = c == 0u ? t.q0.x : c == 1u ? t.q0.w : t.q1.z;
    const float py = c == 0u ? t.q0.y : c == 1u ? t.q1.x : t.q1.w;
    const float pz = c == 0u ? t.q0.z : c == 1u ? t.q1.y : t.q2.x;
    float x, y, d;
    project_vertex(frame, px, py, pz, tile, v, x, y, d);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        p.x[k] = __shfl_sync(0xffffffffu, x, k, kLanes);
        p.y[k] = __shfl_sync(0xffffffffu, y, k, kLanes);
        p.d[k] = __shfl_sync(0xffffffffu, d, k, kLanes);
    }
}

// edge() of facetrtcore.cpp:1287-1290, argument order kept.
__device__ __forceinline__ float edgef(float ax, float ay, float bx, float by, float px, float py)
{
    return (px - ax) * (by - ay) - (py - ay) * (bx - ax);
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
    float m = a;
    if (b < m) m = b;
    if (c < m) m = c;
    return m;
}
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float m = a;
    if (m < b) m = b;
    if (m < c) m = c;
    return m;
}

struct Bbox {
    int x0, x1, y0, y1;
    float area;
    bool valid;
};

// facetrtcore.cpp:1292-1308
__device__ __forceinline__ Bbox triangle_bbox(const RasterFrame& frame, const Projected& p)
{
    Bbox b;
    b.area = edgef(p.x[0], p.y[0], p.x[1], p.y[1], p.x[2], p.y[2]);
    b.valid = !(fabsf(b.area) < 1.0e-8f);
    b.x0 = max(0, int(floorf(min3(p.x[0], p.x[1], p.x[2]))));
    b.x1 = min(int(frame.width) - 1, int(ceilf(max3(p.x[0], p.x[1], p.x[2]))));
    b.y0 = max(0, int(floorf(min3(p.y[0], p.y[1], p.y[2]))));
    b.y1 = min(int(frame.height) - 1, int(ceilf(max3(p.y[0], p.y[1], p.y[2]))));
    if (b.x1 < b.x0 || b.y1 < b.y0) b.valid = false;
    return b;
}

// Inclusive coverage and depth at one pixel centre (facetrtcore.cpp:1309-1332).
__device__ __forceinline__ bool cover(const Projected& p, float area, int x, int y, float& depth)
{
    const float px = float(x) + 0.5f;
    const float py = float(y) + 0.5f;
    const float w0 = edgef(p.x[1], p.y[1], p.x[2], p.y[2], px, py);
    const float w1 = edgef(p.x[2], p.y[2], p.x[0], p.y[0], px, py);
    const float w2 = edgef(p.x[0], p.y[0], p.x[1], p.y[1], px, py);
    const bool inside = area > 0.0f ? (w0 >= 0.0f && w1 >= 0.0f && w2 >= 0.0f)
                                    : (w0 <= 0.0f && w1 <= 0.0f && w2 <= 0.0f);
    if (!inside) return false;
    const float inv = 1.0f / area;
    depth = (w0 * p.d[0] + w1 * p.d[1] + w2 * p.d[2]) * inv;
    return true;
}

__device__ __forceinline__ bool inside(const Projected& p, float area, int x, int y)
{
    float unused;
    return cover(p, area, x, y, unused);
}

struct Pool {
    uint32_t* heads;                 // per pixel: 1 + its newest node, or 0
    uint4* nodes;                    // depth bits, key, the older node (1 + index, or 0)
    uint64_t capacity;
    unsigned long long* used;        // also counts what found no room
    // kNearest, the sun pass: heads count a pixel's fragments, and this keeps the
    // chain key of its first one.  (From lists, a thread walked its pixel's nodes
    // for it.  With / without them: 900 sheets over 128 x 128 pixels 1,474 / 93 us,
    // 20,000 leaves with 0.9 m edges over 1,024 x 1,024 432 / 262, 4,050 facets of
    // terrain 96 / 88, one facet over 64 x 64 88 / 72.)
    unsigned long long* nearest;
};

// A fragment as a number whose order is the chain's: depth, then append order
// (frag_less_stable); the flip bit lies below both.
__device__ __forceinline__ uint64_t chain_key(float depth, uint32_t key)
{
    const uint32_t bits = __float_as_uint(depth + 0.0f);  // -0 is 0
    const uint32_t ordered = bits & 0x80000000u ? ~bits : bits | 0x80000000u;
    return (uint64_t(ordered) << 32) | uint64_t((key << 1) | (key >> 31));
}

template <bool kNearest>
__device__ __forceinline__ void put(const Pool& pool, size_t pix, uint64_t slot, float depth,
                                    uint32_t key)
{
    if (kNearest) {
        atomicMin(&pool.nearest[pix], (unsigned long long)chain_key(depth, key));
        atomicAdd(&pool.heads[pix], 1u);
        return;
    }
    if (slot >= pool.capacity) return;
    const uint32_t older = atomicExch(&pool.heads[pix], uint32_t(slot) + 1u);
    pool.nodes[slot] = make_uint4(__float_as_uint(depth), key, older, 0u);
}

// Room in the pool for `mine` fragments of each warp of the block, one atomic
// per block (a single counter takes about one atomic a clock).  All threads
// call; `mine` is the warp's.
struct Room {
    uint32_t warp[8];
    unsigned long long base;
};
__device__ __forceinline__ uint64_t take_room(Room& r, uint32_t mine, unsigned long long* counter)
{
    const uint32_t warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31u) == 0u) r.warp[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
        for (int w = 0; w < 8; ++w) all += r.warp[w];
        r.base = all ? atomicAdd(counter, (unsigned long long)all) : 0ull;
    }
    __syncthreads();
    uint64_t base = r.base;
    for (uint32_t w = 0; w < warp; ++w) base += r.warp[w];
    return base;
}

__device__ __forceinline__ uint32_t scan_inclusive(uint32_t v)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31u) >= uint32_t(o)) v += y;
    }
    return v;
}

// A triangle, tile and direction (blockIdx.y) per thread.  Boxes of up to
// kSmallPixels pixels are done here: one thread walking a box of hundreds waits
// for as many atomics in turn.  Larger ones are listed, for some lanes each
// from the front of `jobs` and for whole blocks from its back.
// Bound by instructions (69 % of the issue slots; nine IEEE divides to project
// a triangle): 351 us for the 8 M triangles of the forest, where counting and
// filling in two passes took 268 + 448.
template <bool kNearest>
__global__ void __launch_bounds__(256) k_raster(const __grid_constant__ Scene scene,
                                                const float4* __restrict__ planes, uint32_t per_dir,
                                                Pool pool, uint32_t* jobs, uint32_t items,
                                                RasterStats* stats, uint32_t* frags)
{
    start_next();
    __shared__ Room room;
    __shared__ uint32_t warp_mid[8], warp_big[8], base_mid, base_big;
    const uint32_t w = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31u,
                   warp = threadIdx.x >> 5;
    const uint32_t item = blockIdx.y * per_dir + w;
    Projected p;
    Bbox b;
    b.valid = false;
    uint32_t box = 0, side = 0, key = 0, mask = 0;
    if (w < per_dir) {
        const RasterFrame& frame = scene.frame;
        const uint32_t tile = frame.tiles == 1u ? 0u : w / frame.facets;
        const uint32_t facet = w - tile * frame.facets;
        const Facet t = load_facet(frame, planes, facet);
        const uint32_t flip = facing(t, scene.views[blockIdx.y]);
        project(frame, t, tile, scene.views[blockIdx.y], p);
        b = triangle_bbox(frame, p);
        key = w | (flip << 31);
        side = 2u * facet + flip;
        if (b.valid) box = uint32_t(b.x1 - b.x0 + 1) * uint32_t(b.y1 - b.y0 + 1);
        if (box <= kSmallPixels && b.valid) {
            uint32_t bit = 1u;
            for (int y = b.y0; y <= b.y1; ++y)
                for (int x = b.x0; x <= b.x1; ++x, bit <<= 1)
                    if (inside(p, b.area, x, y)) mask |= bit;
        }
    }
    const uint32_t n = __popc(mask);
    if (n && frags) atomicAdd(&frags[side], n);
    const uint32_t incl = scan_inclusive(n);
    const uint32_t mid = __ballot_sync(0xffffffffu, box > kSmallPixels && box <= kBigPixels);
    const uint32_t big = __ballot_sync(0xffffffffu, box > kBigPixels);
    if (lane == 0) {
        warp_mid[warp] = __popc(mid);
        warp_big[warp] = __popc(big);
    }
    uint64_t slot = take_room(room, __shfl_sync(0xffffffffu, incl, 31), pool.used) + (incl - n);
    if (threadIdx.x < 2) {
        const uint32_t* from = threadIdx.x ? warp_big : warp_mid;
        uint32_t all = 0;
        for (int k = 0; k < 8; ++k) all += from[k];
        if (all) all = atomicAdd(threadIdx.x ? &stats->big : &stats->mid, all);
        (threadIdx.x ? base_big : base_mid) = all;
    }
    if (mask) {
        const uint32_t width = scene.frame.width;
        const size_t plane = size_t(blockIdx.y) * width * scene.frame.height;
        for (int y = b.y0; y <= b.y1; ++y) {
            for (int x = b.x0; x <= b.x1; ++x, mask >>= 1) {
                if (!(mask & 1u)) continue;
                float depth;
                cover(p, b.area, x, y, depth);
                put<kNearest>(pool, plane + size_t(y) * width + size_t(x), slot++, depth, key);
            }
        }
    }
    __syncthreads();
    if (box <= kSmallPixels) return;
    const bool whole = box > kBigPixels;
    const uint32_t before = (whole ? big : mid) & ((1u << lane) - 1u);
    uint32_t at = (whole ? base_big : base_mid) + uint32_t(__popc(before));
    for (uint32_t k = 0; k < warp; ++k) at += whole ? warp_big[k] : warp_mid[k];
    jobs[whole ? items - 1u - at : at] = item;
}

// kLanes lanes' share of a listed triangle: pixels [first, first + count) of
// its box, at most 32 kLanes, so that a lane's covered ones are the bits of a
// word.  Called by all threads of the block (count 0 where there is none).
// The atomics of four steps are in flight together.
template <uint32_t kLanes, bool kNearest>
__device__ __forceinline__ void raster_span(const Projected& p, const Bbox& b, size_t plane,
                                            uint32_t width, uint32_t key, uint32_t first, uint32_t count,
                                            const Pool& pool, Room& room, uint32_t* count_at)
{
    const uint32_t lane = threadIdx.x & 31u, sub = lane % kLanes;
    const uint32_t bw = count ? uint32_t(b.x1 - b.x0 + 1) : 1u;
    const uint32_t steps = (count + kLanes - 1u) / kLanes;
    const uint32_t col0 = (first + sub) % bw, row0 = (first + sub) / bw;
    const uint32_t step_x = kLanes % bw, step_y = kLanes / bw;
    uint32_t mask = 0;
    uint32_t cx = col0, cy = row0;
    for (uint32_t r = 0; r < steps; ++r) {
        if (r * kLanes + sub < count && inside(p, b.area, b.x0 + int(cx), b.y0 + int(cy)))
            mask |= 1u << r;
        cx += step_x;
        cy += step_y;
        if (cx >= bw) {
            cx -= bw;
            ++cy;
        }
    }
    __syncwarp();
    uint32_t n = __popc(mask);
#pragma unroll
    for (uint32_t o = 1; o < kLanes; o <<= 1) n += __shfl_xor_sync(0xffffffffu, n, int(o));
    if (sub == 0 && n && count_at) atomicAdd(count_at, n);
#pragma unroll
    for (uint32_t o = kLanes; o < 32u; o <<= 1) n += __shfl_xor_sync(0xffffffffu, n, int(o));
    uint64_t slot = take_room(room, n, pool.used);
    const uint32_t most = __reduce_max_sync(0xffffffffu, steps);
    cx = col0;
    cy = row0;
    for (uint32_t r = 0; r < most; r += 4) {
        uint32_t older[4];
        float depth[4];
        uint64_t at[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const bool on = r + k < steps && (mask >> (r + k)) & 1u;
            const uint32_t lanes = __ballot_sync(0xffffffffu, on);
            at[k] = on ? slot + uint32_t(__popc(lanes & ((1u << lane) - 1u))) : ~0ull;
            slot += uint32_t(__popc(lanes));
            if (kNearest) {
                if (on) {
                    const int x = b.x0 + int(cx), y = b.y0 + int(cy);
                    cover(p, b.area, x, y, depth[k]);
                    put<true>(pool, plane + size_t(y) * width + size_t(x), 0, depth[k], key);
                }
            } else if (at[k] < pool.capacity) {
                const int x = b.x0 + int(cx), y = b.y0 + int(cy);
                cover(p, b.area, x, y, depth[k]);
                older[k] = atomicExch(&pool.heads[plane + size_t(y) * width + size_t(x)],
                                      uint32_t(at[k]) + 1u);
            }
            cx += step_x;
            cy += step_y;
            if (cx >= bw) {
                cx -= bw;
                ++cy;
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
            if (!kNearest && at[k] < pool.capacity)
                pool.nodes[at[k]] = make_uint4(__float_as_uint(depth[k]), key, older[k], 0u);
    }
    __syncthreads();  // room is free again
}

struct Job {
    Projected p;
    Bbox b;
    size_t plane;
    uint32_t key, side;
};
template <uint32_t kLanes>
__device__ __forceinline__ void load_job(const Scene& scene, const float4* planes, uint32_t per_dir,
                                         uint32_t item, Job& j)
{
    const uint32_t dir = item / per_dir, w = item - dir * per_dir;
    const RasterFrame& frame = scene.frame;
    const uint32_t tile = w / frame.facets, facet = w - tile * frame.facets;
    const Facet t = load_facet(frame, planes, facet);
    const uint32_t flip = facing(t, scene.views[dir]);
    project_lanes<kLanes>(frame, t, tile, scene.views[dir], j.p);
    j.b = triangle_bbox(frame, j.p);
    j.plane = size_t(dir) * frame.width * frame.height;
    j.key = w | (flip << 31);
    j.side = 2u * facet + flip;
}

// Bound by instructions and the latency of its rounds (issue 57 %): 323 us for
// the forest's 0.8 M ground triangles, 190 us for the terrain's 164,000, which
// took 160 + 495 in two passes of a thread each.
template <uint32_t kLanes, bool kNearest>
__global__ void __launch_bounds__(256) k_raster_mid(const __grid_constant__ Scene scene,
                                                    const float4* __restrict__ planes,
                                                    uint32_t per_dir, Pool pool,
                                                    const uint32_t* jobs,
                                                    const uint32_t* job_count,
                                                    uint32_t* frags)
{
    start_next();
    wait_for_previous();
    __shared__ Room room;
    const uint32_t count = *job_count;
    constexpr uint32_t kJobs = 256 / kLanes, kSpan = 32 * kLanes;
    for (uint32_t k = blockIdx.x * kJobs; k < count; k += gridDim.x * kJobs) {
        const uint32_t mine = k + threadIdx.x / kLanes;
        Job j;
        load_job<kLanes>(scene, planes, per_dir, jobs[mine < count ? mine : k], j);
        const uint32_t box = mine < count ? uint32_t(j.b.x1 - j.b.x0 + 1) *
                                                uint32_t(j.b.y1 - j.b.y0 + 1) : 0u;
        for (uint32_t first = 0; __syncthreads_or(int(first < box)); first += kSpan)
            raster_span<kLanes, kNearest>(j.p, j.b, j.plane, scene.frame.width, j.key, first,
                                first < box ? min(box - first, kSpan) : 0u, pool, room,
                                frags ? frags + j.side : nullptr);
    }
}

// Triangles with boxes above kBigPixels.  A few share the grid, several blocks to
// each; with more than the grid has warps, a warp takes one.  40 directions of 20,000
// facets with boxes of some 3,000 pixels: 3.4 ms, 24.4 where every 16th block took
// whole triangles and the others looked for parts beyond 8,192 pixels; a sheet over
// the whole frame takes 16 blocks or more as before.
template <bool kNearest>
__global__ void __launch_bounds__(256) k_raster_big(const __grid_constant__ Scene scene,
                                                    const float4* __restrict__ planes,
                                                    uint32_t per_dir, Pool pool,
                                                    const uint32_t* jobs_end,
                                                    const uint32_t* job_count,
                                                    uint32_t* frags)
{
    start_next();
    wait_for_previous();
    __shared__ Room room;
    const uint32_t count = *job_count, warp = threadIdx.x >> 5;
    if (!count) return;
    // spans of a job for each `stride` pixels from `first`, in step with the block
    auto draw = [&](uint32_t item, bool on, uint32_t first, uint32_t stride) {
        Job j;
        load_job<32>(scene, planes, per_dir, item, j);
        const uint32_t box =
            on ? uint32_t(j.b.x1 - j.b.x0 + 1) * uint32_t(j.b.y1 - j.b.y0 + 1) : 0u;
        for (; __syncthreads_or(int(first < box)); first += stride)
            raster_span<32, kNearest>(j.p, j.b, j.plane, scene.frame.width, j.key, first < box ? first : 0u,
                            first < box ? min(box - first, kBigPixels) : 0u, pool, room,
                            frags ? frags + j.side : nullptr);
    };
    if (count >= 8u * gridDim.x) {  // a warp each
        for (uint32_t k = blockIdx.x * 8u; k < count; k += gridDim.x * 8u)
            draw(*(jobs_end - 1 - min(k + warp, count - 1u)), k + warp < count, 0u, kBigPixels);
    } else {  // several blocks, or one, to each
        const uint32_t share = max(1u, gridDim.x / count), part = blockIdx.x % share;
        for (uint32_t k = blockIdx.x / share; k < count; k += (gridDim.x + share - 1u) / share)
            draw(*(jobs_end - 1 - k), true, (part * 8u + warp) * kBigPixels, share * 8u * kBigPixels);
    }
}

// Both sides of a facet have the denominator of all its fragments.
__global__ void k_denominators(uint32_t facets, const uint2* __restrict__ frags,
                               uint2* __restrict__ denom)
{
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= facets) return;
    const uint32_t n = frags[f].x + frags[f].y;
    denom[f] = make_uint2(n, n);
}

// ---- per-pixel ordering ------------------------------------------------------
struct Frag {
    float depth;
    uint32_t key;  // append order | flip << 31
};

__device__ __forceinline__ bool frag_less(const Frag& a, const Frag& b) { return a.depth < b.depth; }

__device__ __forceinline__ bool frag_less_stable(const Frag& a, const Frag& b)
{
    return a.depth < b.depth || (a.depth == b.depth && (a.key & kKeyMask) < (b.key & kKeyMask));
}

__device__ void sort_by_append_order(Frag* f, int n)
{
    for (int i = 1; i < n; ++i) {
        const Frag v = f[i];
        int j = i;
        while (j > 0 && (f[j - 1].key & kKeyMask) > (v.key & kKeyMask)) {
            f[j] = f[j - 1];
            --j;
        }
        f[j] = v;
    }
}

// GCC libstdc++ std::sort, restated (see the oracle for the same steps):
// introsort with median-of-three, unguarded partition, heap-sort fallback at
// depth 2*floor(log2 n), final insertion sort with threshold 16.
// The bounds checks below never trigger when the introsort invariants hold
// (a smaller-or-equal element precedes every unguarded insertion, the
// partition scans stop inside the range); they only keep a wrong input from
// walking out of the local array.
__device__ void unguarded_linear_insert(Frag* f, int last)
{
    const Frag v = f[last];
    int next = last - 1;
    while (next >= 0 && frag_less(v, f[next])) {
        f[last] = f[next];
        last = next;
        --next;
    }
    f[last] = v;
}

__device__ void insertion_sort(Frag* f, int first, int last)
{
    if (first == last) return;
    for (int i = first + 1; i != last; ++i) {
        if (frag_less(f[i], f[first])) {
            const Frag v = f[i];
            for (int k = i; k > first; --k) f[k] = f[k - 1];
            f[first] = v;
        } else {
            unguarded_linear_insert(f, i);
        }
    }
}

__device__ void adjust_heap(Frag* first, int hole, int len, Frag value)
{
    const int top = hole;
    int child = hole;
    while (child < (len - 1) / 2) {
        child = 2 * (child + 1);
        if (frag_less(first[child], first[child - 1])) child--;
        first[hole] = first[child];
        hole = child;
    }
    if ((len & 1) == 0 && child == (len - 2) / 2) {
        child = 2 * (child + 1);
        first[hole] = first[child - 1];
        hole = child - 1;
    }
    int parent = (hole - 1) / 2;
    while (hole > top && frag_less(first[parent], value)) {
        first[hole] = first[parent];
        hole = parent;
        parent = (hole - 1) / 2;
    }
    first[hole] = value;
}

__device__ void heap_sort(Frag* first, int len)
{
    if (len >= 2) {
        int parent = (len - 2) / 2;
        for (;;) {
            adjust_heap(first, parent, len, first[parent]);
            if (parent == 0) break;
            parent--;
        }
    }
    while (len > 1) {
        --len;
        const Frag v = first[len];
        first[len] = first[0];
        adjust_heap(first, 0, len, v);
    }
}

__device__ __forceinline__ void fswap(Frag& a, Frag& b)
{
    const Frag t = a;
    a = b;
    b = t;
}

__device__ void median_to_first(Frag* f, int result, int a, int b, int c)
{
    if (frag_less(f[a], f[b])) {
        if (frag_less(f[b], f[c])) fswap(f[result], f[b]);
        else if (frag_less(f[a], f[c])) fswap(f[result], f[c]);
        else fswap(f[result], f[a]);
    } else if (frag_less(f[a], f[c])) fswap(f[result], f[a]);
    else if (frag_less(f[b], f[c])) fswap(f[result], f[c]);
    else fswap(f[result], f[b]);
}

__device__ int unguarded_partition(Frag* f, int first, int last, int pivot)
{
    const int lo = first, hi = last;
    for (;;) {
        while (first < hi - 1 && frag_less(f[first], f[pivot])) ++first;
        --last;
        while (last > lo && frag_less(f[pivot], f[last])) --last;
        if (!(first < last)) return first;
        fswap(f[first], f[last]);
        ++first;
    }
}

__device__ void std_sort_by_depth(Frag* f, int n)
{
    if (n <= 1) return;
    if (n <= 16) {
        insertion_sort(f, 0, n);
        return;
    }
    int lg = 0;
    while ((1 << (lg + 1)) <= n) ++lg;
    // introsort loop with an explicit stack of pending right-hand ranges
    int stack_first[64], stack_last[64], stack_depth[64];
    int sp = 0;
    stack_first[sp] = 0;
    stack_last[sp] = n;
    stack_depth[sp] = 2 * lg;
    ++sp;
    while (sp > 0) {
        --sp;
        const int first = stack_first[sp];
        int last = stack_last[sp];
        int depth = stack_depth[sp];
        // The recursion of the reference handles (cut, last) before the
        // left part; ranges are disjoint, so order between them does not
        // change the result.
        while (last - first > 16) {
            if (depth == 0) {
                heap_sort(f + first, last - first);
                break;
            }
            --depth;
            const int mid = first + (last - first) / 2;
            median_to_first(f, first, first + 1, mid, last - 1);
            const int cut = unguarded_partition(f, first + 1, last, first);
            if (sp < 64) {
                stack_first[sp] = cut;
                stack_last[sp] = last;
                stack_depth[sp] = depth;
                ++sp;
            }
            last = cut;
        }
    }
    insertion_sort(f, 0, 16);
    for (int i = 16; i < n; ++i) unguarded_linear_insert(f, i);
}

__device__ __forceinline__ void order_chain(Frag* f, int n)
{
    if (n <= 16) {
        // libstdc++ sorts <= 16 elements by insertion sort, which is stable:
        // the result is sorted by (depth, append order) whatever the load order.
        for (int i = 1; i < n; ++i) {
            const Frag v = f[i];
            int j = i;
            while (j > 0 && frag_less_stable(v, f[j - 1])) {
                f[j] = f[j - 1];
                --j;
            }
            f[j] = v;
        }
    } else {
        sort_by_append_order(f, n);
        std_sort_by_depth(f, n);
    }
}

__device__ __forceinline__ uint32_t frag_side(uint32_t key, uint32_t facets)
{
    const uint32_t order = key & kKeyMask;
    return 2u * (order % facets) + (key >> 31);
}

// Room for `mine` pairs of each lane, one atomic a warp (one counter takes about
// one atomic a clock).
__device__ __forceinline__ unsigned long long take_pairs(uint32_t mine,
                                                         unsigned long long* pair_count)
{
    const uint32_t incl = scan_inclusive(mine);
    unsigned long long base = 0;
    if ((threadIdx.x & 31u) == 31u && incl) base = atomicAdd(pair_count, (unsigned long long)incl);
    return __shfl_sync(0xffffffffu, base, 31) + (incl - mine);
}

// Emit sky counts and adjacent pairs of an ordered chain
// (facetrtcore.cpp:1374-1392; visibility_resolve.comp:102-116).  Called by whole
// warps (n = 0: no chain), which take their room in `pairs` with one atomic.
__device__ void emit_chain(const Frag* f, int n, uint32_t facets, uint32_t* sky, uint64_t* pairs,
                           unsigned long long* pair_count, int side_bits)
{
    if (n > 0) {
        atomicAdd(&sky[frag_side(f[0].key, facets)], 1u);
        atomicAdd(&sky[frag_side(f[n - 1].key, facets) ^ 1u], 1u);
    }
    uint32_t np = 0;
    for (int i = 0; i + 1 < n; ++i) {
        const uint32_t a = frag_side(f[i].key, facets) ^ 1u;
        const uint32_t b = frag_side(f[i + 1].key, facets);
        if ((a >> 1) != (b >> 1)) ++np;
    }
    __syncwarp();
    unsigned long long base = take_pairs(np, pair_count);
    uint32_t k = 0;
    for (int i = 0; i + 1 < n; ++i) {
        const uint32_t a = frag_side(f[i].key, facets) ^ 1u;
        const uint32_t b = frag_side(f[i + 1].key, facets);
        if ((a >> 1) == (b >> 1)) continue;
        const uint64_t lo = a < b ? a : b, hi = a < b ? b : a;
        pairs[base + k] = (lo << side_bits) | hi;
        ++k;
    }
}

__device__ __forceinline__ uint64_t chain_key(const uint4& node)
{
    return chain_key(__uint_as_float(node.x), node.y);
}
__device__ __forceinline__ uint32_t key_side(uint64_t k, uint32_t facets, uint32_t tiles)
{
    const uint32_t low = uint32_t(k);  // the side itself where there is one tile
    return tiles == 1u ? low : 2u * ((low >> 1) % facets) + (low & 1u);
}

__device__ __forceinline__ void order2(uint64_t& a, uint64_t& b)
{
    const uint64_t lo = a < b ? a : b, hi = a < b ? b : a;
    a = lo;
    b = hi;
}

// The run of lanes with the same side that this lane begins: its length, or 0
// where it begins none.  Neighbouring pixels mostly show one side, so that a
// count takes one atomic per run.
__device__ __forceinline__ uint32_t side_run(uint32_t side, bool on)
{
    const uint32_t lane = threadIdx.x & 31u, key = on ? side : 0xffffffffu;
    const uint32_t left = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = lane == 0u || left != key;
    const uint32_t later = __ballot_sync(0xffffffffu, head) & (0xfffffffeu << lane);
    return head && on ? (later ? uint32_t(__ffs(int(later)) - 1) : 32u) - lane : 0u;
}
__device__ __forceinline__ void add_sides(uint32_t* count, uint32_t side, bool on)
{
    const uint32_t run = side_run(side, on);
    if (run) atomicAdd(&count[side], run);
}

// The longest chain that a thread has met.
__device__ __forceinline__ void note_longest(RasterStats* stats, uint32_t n)
{
    const uint32_t most = __reduce_max_sync(0xffffffffu, n);
    if ((threadIdx.x & 31u) == 0u && most > *const_cast<volatile uint32_t*>(&stats->max_chain))
        atomicMax(&stats->max_chain, most);
}

// The block's 2,048 pixels, those that hold fragments packed into `queue`
// (three quarters of the pixels are empty, and whole threads with them).
struct Covered {
    uint32_t queue[2048];
    uint32_t warp[8];
};
__device__ __forceinline__ uint32_t gather_covered(const uint32_t* heads, Covered& c)
{
    const uint4* h = reinterpret_cast<const uint4*>(heads) + size_t(blockIdx.x) * 512 + threadIdx.x;
    const uint4 a = __ldcs(h), b = __ldcs(h + 256);
    const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t n = 0;  // both halves' counts, 16 bits each
#pragma unroll
    for (int k = 0; k < 8; ++k) n += v[k] ? (k < 4 ? 1u : 0x10000u) : 0u;
    const uint32_t incl = scan_inclusive(n), warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31u) == 31u) c.warp[warp] = incl;
    __syncthreads();
    uint32_t before = incl - n, all = 0;
    for (uint32_t w = 0; w < 8; ++w) {
        if (w < warp) before += c.warp[w];
        all += c.warp[w];
    }
    uint32_t at = before & 0xffffu;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k == 4) at = (all & 0xffffu) + (before >> 16);
        if (v[k]) c.queue[at++] = v[k];
    }
    __syncthreads();
    return (all & 0xffffu) + (all >> 16);
}

// Pixels with longer chains than kFast, by length: for networks of 16 and of 32
// keys, and the rest.
struct Lists {
    uint2 *at16, *at32, *rest;  // {1 + the newest node, fragments}
};

// A thread per covered pixel, chains of at most kFast fragments ordered in
// registers (most have one); longer ones are listed.  The
// block's pairs wait in shared memory and leave together: with one atomic and a
// barrier per 256 pixels this took 208 us for the terrain's 42 M pixels and 252
// for the forest's, now 171 and 181; 64 fragments of local memory for every
// pixel and two denominator atomics per fragment took 871 and 460.  Bound by
// instructions and the two loads in a row, pixel and fragment.
constexpr uint32_t kHeldPairs = 1024;
__global__ void __launch_bounds__(256) k_resolve_graph(
    uint32_t facets, uint32_t tiles, const uint32_t* __restrict__ heads, const uint4* __restrict__ nodes, uint32_t cap,
    uint32_t* sky, uint64_t* pairs, unsigned long long* pair_count, int side_bits, Lists lists,
    RasterStats* stats)
{
    start_next();
    __shared__ Covered c;
    __shared__ uint64_t held[kHeldPairs];
    __shared__ uint32_t held_count, held_end;
    __shared__ unsigned long long out;
    if (threadIdx.x == 0) held_count = 0;
    const uint32_t covered = gather_covered(heads, c);
    if (!covered) return;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t longest = 0;
    for (uint32_t first = threadIdx.x & ~31u; first < covered; first += 256) {
        const uint32_t head = first + lane < covered ? c.queue[first + lane] : 0u;
        uint64_t k[kFast];
        uint32_t n = 0, next = 0;
        k[0] = ~0ull;
        if (head) {
            const uint4 node = __ldcs(nodes + (head - 1u));
            k[0] = chain_key(node);
            next = node.z;
            n = 1;
        }
        if (!__any_sync(0xffffffffu, next != 0u)) {
            const uint32_t side = key_side(k[0], facets, tiles), run = side_run(side, n != 0u);
            if (run) {
                atomicAdd(&sky[side], run);
                atomicAdd(&sky[side ^ 1u], run);
            }
            if (n > cap) atomicAdd(&stats->overflow, (unsigned long long)(n - cap));
            longest = max(longest, n);
            continue;
        }
#pragma unroll
        for (int q = 1; q < kFast; ++q) {
            k[q] = ~0ull;
            if (next) {
                const uint4 node = __ldcs(nodes + (next - 1u));
                k[q] = chain_key(node);
                next = node.z;
                ++n;
            }
        }
        const bool is_long = next != 0u;
        while (next) {
            next = nodes[next - 1u].z;
            ++n;
        }
        if (__any_sync(0xffffffffu, is_long)) {
            const uint32_t which = n <= 16u ? 0u : n <= 32u ? 1u : 2u;
#pragma unroll
            for (uint32_t l = 0; l < 3; ++l) {  // one atomic a warp and list
                const uint32_t lanes = __ballot_sync(0xffffffffu, is_long && which == l);
                if (!lanes) continue;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&stats->listed[l], uint32_t(__popc(lanes)));
                at = __shfl_sync(0xffffffffu, at, 0) + uint32_t(__popc(lanes & ((1u << lane) - 1u)));
                if (lanes >> lane & 1u)
                    (l == 0 ? lists.at16 : l == 1 ? lists.at32 : lists.rest)[at] = make_uint2(head, n);
            }
        }
        if (n > cap) atomicAdd(&stats->overflow, (unsigned long long)(n - cap));
        longest = max(longest, n);
        if (n > uint32_t(kFast)) n = 0;
        const uint32_t most = __reduce_max_sync(0xffffffffu, n);
        // Batcher's networks for 2, 4 and 8 keys
        order2(k[0], k[1]);
        if (most > 2u) {
            order2(k[2], k[3]);
            order2(k[0], k[2]);
            order2(k[1], k[3]);
            order2(k[1], k[2]);
        }
        if (most > 4u) {
            order2(k[4], k[5]);
            order2(k[6], k[7]);
            order2(k[4], k[6]);
            order2(k[5], k[7]);
            order2(k[5], k[6]);
            order2(k[0], k[4]);
            order2(k[1], k[5]);
            order2(k[2], k[6]);
            order2(k[3], k[7]);
            order2(k[2], k[4]);
            order2(k[3], k[5]);
            order2(k[1], k[2]);
            order2(k[3], k[4]);
            order2(k[5], k[6]);
        }
        uint32_t side[kFast], mine = 0;
        side[0] = key_side(k[0], facets, tiles);
        uint32_t last = side[0];
#pragma unroll
        for (int q = 1; q < kFast; ++q) {
            if (uint32_t(q) >= most) break;
            side[q] = key_side(k[q], facets, tiles);
            if (uint32_t(q) < n) {
                last = side[q];
                if ((side[q - 1] >> 1) != (side[q] >> 1)) ++mine;
            }
        }
        add_sides(sky, side[0], n != 0u);
        add_sides(sky, last ^ 1u, n != 0u);
        if (!__any_sync(0xffffffffu, mine != 0u)) continue;
        const uint32_t incl = scan_inclusive(mine);
        const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&held_count, all);
        base = __shfl_sync(0xffffffffu, base, 0);
        uint64_t* to = held + (base + incl - mine);
        if (base + all > kHeldPairs) {
            // No room: straight out.  All later requests end here too, and the
            // first of them marks the end of what is held.
            if (lane == 0 && base <= kHeldPairs) held_end = base;
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(pair_count, (unsigned long long)all);
            to = pairs + __shfl_sync(0xffffffffu, at, 0) + (incl - mine);
        }
#pragma unroll
        for (int q = 1; q < kFast; ++q) {
            if (uint32_t(q) >= most) break;
            if (uint32_t(q) >= n || (side[q - 1] >> 1) == (side[q] >> 1)) continue;
            const uint32_t a = side[q - 1] ^ 1u, b = side[q];
            const uint64_t lo = a < b ? a : b, hi = a < b ? b : a;
            *to++ = (lo << side_bits) | hi;
        }
    }
    note_longest(stats, longest);
    __syncthreads();
    const uint32_t keep = held_count > kHeldPairs ? held_end : held_count;
    if (threadIdx.x == 0 && keep) out = atomicAdd(pair_count, (unsigned long long)keep);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < keep; i += 256) pairs[out + i] = held[i];
}

// Batcher's odd-even merge sort of N keys, from merges of P with strides of Q on.
template <int N, int P, int Q>
__device__ __forceinline__ void network(uint64_t (&k)[N])
{
    constexpr int first = Q % P;
#pragma unroll
    for (int i = first; i < N - Q; ++i)
        if ((i - first) / Q % 2 == 0 && i / (2 * P) == (i + Q) / (2 * P)) order2(k[i], k[i + Q]);
    if constexpr (Q > 1) network<N, P, Q / 2>(k);
    else if constexpr (2 * P < N) network<N, 2 * P, 2 * P>(k);
}

// Listed pixels with at most N fragments, a thread each, ordered by Batcher's
// network in registers, without local memory and in step (insertion sorts in local
// memory kept 10 of 32 lanes busy).  40 directions of 60,000 facets of some 0.4 m:
// chains of 9 to 16 take 1.15 ms and of 17 to 32 0.39, 9.5 by sorts in local memory
// and an atomic for each pixel's pairs.  Bound by the loads along the chain.  Where two of more than 16 fragments
// share a depth, std::sort's order is not the append order, and the pixel goes to the
// rest's list.
template <int N>
__global__ void __launch_bounds__(128) k_resolve_network(
    uint32_t facets, uint32_t tiles, const uint4* __restrict__ nodes, const uint2* list,
    const uint32_t* count, uint32_t* sky, uint64_t* pairs, unsigned long long* pair_count,
    int side_bits, uint2* rest, uint32_t* rest_count)
{
    start_next();
    wait_for_previous();
    const uint32_t listed = *count;
    for (uint32_t j0 = blockIdx.x * 128 + (threadIdx.x & ~31u); j0 < listed; j0 += gridDim.x * 128) {
        const uint32_t j = j0 + (threadIdx.x & 31u);
        const uint2 mine = j < listed ? list[j] : make_uint2(0u, 0u);
        uint32_t next = mine.x, n = mine.y;
        uint64_t k[N];
#pragma unroll
        for (int q = 0; q < N; ++q) {
            k[q] = ~0ull;
            if (next) {
                const uint4 node = __ldcs(nodes + (next - 1u));
                k[q] = chain_key(node);
                next = node.z;
            }
        }
        __syncwarp();
        network<N, 1, 1>(k);
        if (N > 16) {
            bool tie = false;
#pragma unroll
            for (int q = 1; q < N; ++q) tie |= uint32_t(q) < n && k[q] >> 32 == k[q - 1] >> 32;
            if (tie) {
                rest[atomicAdd(rest_count, 1u)] = mine;
                n = 0;
            }
            __syncwarp();
        }
        uint32_t before = key_side(k[0], facets, tiles), np = 0;
        const uint32_t nearest = before;
#pragma unroll
        for (int q = 1; q < N; ++q)
            if (uint32_t(q) < n) {
                const uint32_t side = key_side(k[q], facets, tiles);
                np += (before >> 1) != (side >> 1) ? 1u : 0u;
                before = side;
            }
        if (n) {
            atomicAdd(&sky[nearest], 1u);
            atomicAdd(&sky[before ^ 1u], 1u);
        }
        __syncwarp();
        uint64_t* to = pairs + take_pairs(np, pair_count);
        before = nearest;
#pragma unroll
        for (int q = 1; q < N; ++q)
            if (uint32_t(q) < n) {
                const uint32_t side = key_side(k[q], facets, tiles), a = before ^ 1u;
                if ((before >> 1) != (side >> 1))
                    *to++ = (uint64_t(min(a, side)) << side_bits) | max(a, side);
                before = side;
            }
    }
}

// The rest, pixels with more than `above` and at most kCap fragments, a thread
// each, in local memory; chains above kDeepChain are an error.  A list begins with
// its newest fragment, so it is laid out from the back: near the append order that
// long chains are brought into first.
template <uint32_t kCap>
__global__ void __launch_bounds__(64) k_resolve_list(
    uint32_t facets, const uint4* __restrict__ nodes, const uint2* list, uint32_t above, uint32_t* sky,
    uint64_t* pairs, unsigned long long* pair_count, int side_bits, RasterStats* stats)
{
    start_next();
    wait_for_previous();
    const uint32_t listed = stats->listed[2];
    for (uint32_t j0 = blockIdx.x * 64 + (threadIdx.x & ~31u); j0 < listed; j0 += gridDim.x * 64) {
        const uint32_t j = j0 + (threadIdx.x & 31u);
        uint32_t n = j < listed ? list[j].y : 0u;
        if (n > kCap) {
            // (kMidChain: the next launch's)
            if (kCap == kDeepChain) atomicAdd(&stats->capacity_error, 1u);
            n = 0;
        }
        if (n <= above) n = 0;
        if (!__any_sync(0xffffffffu, n != 0u)) continue;
        Frag f[kCap];
        uint32_t next = n ? list[j].x : 0u;
        for (uint32_t k = n; k-- > 0;) {
            const uint4 node = nodes[next - 1u];
            f[k].depth = __uint_as_float(node.x);
            f[k].key = node.y;
            next = node.z;
        }
        order_chain(f, int(n));
        emit_chain(f, int(n), facets, sky, pairs, pair_count, side_bits);
    }
}

// computeCpuSunlit per pixel (facetrtcore.cpp:1448-1466): the nearest fragment
// (first in append order among equal depths) is visible.  (Every fragment
// counts towards its side's total: counted by the raster.)  Bound by reading the
// counts; a warp without fragments reads nothing else.
__global__ void __launch_bounds__(256) k_resolve_sunlit(uint32_t facets, uint32_t tiles,
                                                        const uint32_t* __restrict__ counts,
                                                        const uint64_t* __restrict__ nearest,
                                                        uint64_t npix, uint32_t cap,
                                                        uint32_t* visible, RasterStats* stats)
{
    uint32_t longest = 0;
    const uint64_t stride = uint64_t(gridDim.x) * 256;
    for (uint64_t first = uint64_t(blockIdx.x) * 256 + (threadIdx.x & ~31u); first < npix;
         first += stride) {
        const uint64_t i = first + (threadIdx.x & 31u);
        const uint32_t n = i < npix ? __ldcs(counts + i) : 0u;
        if (!__any_sync(0xffffffffu, n != 0u)) continue;
        const uint64_t best = n ? __ldcs(nearest + i) : ~0ull;
        if (n > cap) atomicAdd(&stats->overflow, (unsigned long long)(n - cap));
        longest = max(longest, n);
        __syncwarp();
        add_sides(visible, key_side(best, facets, tiles), n != 0u);
    }
    note_longest(stats, longest);
}

__global__ void k_fraction(uint32_t S, const uint32_t* total, const uint32_t* visible, float* out)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < S) out[s] = total[s] ? float(visible[s]) / float(total[s]) : 0.0f;
}

}  // namespace

namespace {
unsigned sm_count()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return unsigned(std::max(sms, 1));
}
}  // namespace

namespace {

// The rasters of all directions, into the pool's lists or nearest fragments.
struct RasterPass {
    Scene scene{};
    uint64_t npix = 0, per_dir = 0, items = 0;
    unsigned sms = 0;
    uint32_t* jobs = nullptr;
    float4* planes = nullptr;
    RasterStats* stats = nullptr;
    RasterPass(const facetcu_vertex* d_vertices, const RasterFrame& frame, const RasterView* views,
               uint32_t dir_count, RasterBuffers& rb, cudaStream_t s)
    {
        if (dir_count > kMaxViews)
            throw Error(FACETCU_INVALID_ARGUMENT, "raster chunk exceeds 64 directions");
        scene.frame = frame;
        std::copy(views, views + dir_count, scene.views);
        npix = uint64_t(dir_count) * frame.width * frame.height;
        per_dir = uint64_t(frame.tiles) * frame.facets;
        items = dir_count * per_dir;
        if (items >= (1ull << 32))
            throw Error(FACETCU_OVERFLOW_ERROR, "raster work exceeds 2^32 triangles");
        sms = sm_count();
        jobs = static_cast<uint32_t*>(rb.jobs.reserve(items * 4));
        planes = static_cast<float4*>(rb.planes.reserve(size_t(frame.facets) * 48));
        stats = static_cast<RasterStats*>(rb.stats.reserve(sizeof(RasterStats)));
        k_planes<<<(frame.facets + 255) / 256, 256, 0, s>>>(d_vertices, frame.facets, planes);
        FCU_LAUNCH("k_planes");
    }
    template <bool kNearest>
    void run(const Pool& pool, uint32_t* d_frags, uint32_t dir_count, cudaStream_t s) const
    {
        FCU_CHECK(cudaMemsetAsync(stats, 0, sizeof(RasterStats), s));
        k_raster<kNearest><<<dim3(unsigned((per_dir + 255) / 256), dir_count), 256, 0, s>>>(
            scene, planes, uint32_t(per_dir), pool, jobs, uint32_t(items), stats, d_frags);
        FCU_LAUNCH("k_raster");
        launch_early(k_raster_mid<kMidLanes, kNearest>,
                     unsigned(std::min<uint64_t>((items + 31) / 32, 8u * sms)), 256, 0, s, scene, planes,
                     uint32_t(per_dir), pool, jobs, &stats->mid, d_frags);
        launch_early(k_raster_big<kNearest>, unsigned(std::min<uint64_t>(items * 16, 8u * sms)), 256, 0,
                     s, scene, planes, uint32_t(per_dir), pool, jobs + items, &stats->big, d_frags);
    }
};

void refuse_fragments(const RasterStats& host)
{
    if (host.fragments >= (1ull << 32))
        throw Error(FACETCU_OVERFLOW_ERROR, "more than 2^32 fragments in one raster chunk");
}

}  // namespace

void raster_fragments(const facetcu_vertex* d_vertices, const RasterFrame& frame,
                      const RasterView* views, uint32_t dir_count, RasterBuffers& rb,
                      uint32_t* d_frags, RasterStats& stats, cudaStream_t s)
{
    const RasterPass pass(d_vertices, frame, views, dir_count, rb, s);
    // whole blocks of the resolve
    const uint64_t padded = (pass.npix + kResolvePixels - 1) / kResolvePixels * kResolvePixels;
    uint32_t* heads = static_cast<uint32_t*>(rb.heads.reserve(padded * 4));
    // A pool of one fragment for two pixels to begin with: the forest of
    // 200,000 facets has 0.29 a pixel over the 40 directions, 4,096 facets of
    // terrain 0.25.
    RasterStats host{};
    uint64_t capacity = std::max<uint64_t>(rb.nodes.bytes / 16, pass.npix / 2 + 1);
    for (uint32_t* counted = d_frags;; counted = nullptr) {
        capacity = std::min<uint64_t>(capacity, 0xffffffffull);
        const Pool pool{heads, static_cast<uint4*>(rb.nodes.reserve(capacity * 16)), capacity,
                        &pass.stats->fragments, nullptr};
        FCU_CHECK(cudaMemsetAsync(heads, 0, padded * 4, s));
        pass.run<false>(pool, counted, dir_count, s);
        FCU_CHECK(cudaMemcpyAsync(&host, pass.stats, sizeof(RasterStats), cudaMemcpyDeviceToHost, s));
        FCU_CHECK(cudaStreamSynchronize(s));
        refuse_fragments(host);
        if (host.fragments <= capacity) break;
        capacity = host.fragments;
    }
    stats.fragments = host.fragments;
    stats.big = host.big;
}

void raster_denominators(uint32_t facets, const uint32_t* d_frags, uint32_t* d_denominators,
                         cudaStream_t s)
{
    k_denominators<<<(facets + 255) / 256, 256, 0, s>>>(
        facets, reinterpret_cast<const uint2*>(d_frags), reinterpret_cast<uint2*>(d_denominators));
    FCU_LAUNCH("k_denominators");
}

void raster_resolve_graph(const RasterFrame& frame, uint32_t dir_count, uint32_t chain_cap,
                          RasterBuffers& rb, uint32_t* d_sky, uint64_t* d_pairs,
                          unsigned long long* d_pair_count, int side_bits, RasterStats& stats,
                          cudaStream_t s)
{
    const uint64_t npix = uint64_t(dir_count) * frame.width * frame.height;
    RasterStats* dstats = rb.stats.as<RasterStats>();
    // (pixels of 9, 17 and 17 fragments at least: the last list takes the ties too)
    const size_t room16 = stats.fragments / (kFast + 1) + 1, room32 = stats.fragments / 17 + 1;
    uint2* list = static_cast<uint2*>(rb.list.reserve((room16 + 2 * room32) * 8));
    const Lists lists{list, list + room16, list + room16 + room32};
    const uint4* nodes = rb.nodes.as<uint4>();
    k_resolve_graph<<<unsigned((npix + kResolvePixels - 1) / kResolvePixels), 256, 0, s>>>(
        frame.facets, frame.tiles, rb.heads.as<uint32_t>(), nodes, chain_cap, d_sky, d_pairs,
        d_pair_count, side_bits, lists, dstats);
    FCU_LAUNCH("k_resolve_graph");
    const unsigned list_blocks = 16 * sm_count();
    launch_early(k_resolve_network<16>, list_blocks, 128, 0, s, frame.facets, frame.tiles, nodes,
                 lists.at16, &dstats->listed[0], d_sky, d_pairs, d_pair_count, side_bits, lists.rest,
                 &dstats->listed[2]);
    launch_early(k_resolve_network<32>, list_blocks, 128, 0, s, frame.facets, frame.tiles, nodes,
                 lists.at32, &dstats->listed[1], d_sky, d_pairs, d_pair_count, side_bits, lists.rest,
                 &dstats->listed[2]);
    launch_early(k_resolve_list<kMidChain>, list_blocks, 64, 0, s, frame.facets, nodes, lists.rest, 0u,
                 d_sky, d_pairs, d_pair_count, side_bits, dstats);
    RasterStats host{};
    auto read = [&] {
        FCU_CHECK(cudaMemcpyAsync(&host, dstats, sizeof(RasterStats), cudaMemcpyDeviceToHost, s));
        FCU_CHECK(cudaMemcpyAsync(&stats.pairs, d_pair_count, 8, cudaMemcpyDeviceToHost, s));
        FCU_CHECK(cudaStreamSynchronize(s));
    };
    read();
    if (host.max_chain > kMidChain) {
        // (launched only then: its local memory is a few GB)
        k_resolve_list<kDeepChain><<<list_blocks, 64, 0, s>>>(frame.facets, nodes, lists.rest, kMidChain,
                                                              d_sky, d_pairs, d_pair_count,
                                                              side_bits, dstats);
        FCU_LAUNCH("k_resolve_list");
        read();
    }
    stats.overflow = host.overflow;
    stats.max_chain = host.max_chain;
    stats.capacity_error = host.capacity_error;
}

void raster_sunlit(const facetcu_vertex* d_vertices, const RasterFrame& frame, const RasterView& view,
                   uint32_t chain_cap, RasterBuffers& rb, uint32_t* d_total, uint32_t* d_visible,
                   float* d_fraction, RasterStats& stats, cudaStream_t s)
{
    const RasterPass pass(d_vertices, frame, &view, 1, rb, s);
    uint32_t* counts = static_cast<uint32_t*>(rb.heads.reserve(pass.npix * 4));
    unsigned long long* nearest = static_cast<unsigned long long*>(rb.nodes.reserve(pass.npix * 8));
    FCU_CHECK(cudaMemsetAsync(counts, 0, pass.npix * 4, s));
    FCU_CHECK(cudaMemsetAsync(nearest, 0xff, pass.npix * 8, s));
    pass.run<true>({counts, nullptr, 0, &pass.stats->fragments, nearest}, d_total, 1, s);
    k_resolve_sunlit<<<unsigned(std::min<uint64_t>((pass.npix + 255) / 256, 16u * pass.sms)), 256, 0, s>>>(
        frame.facets, frame.tiles, counts, reinterpret_cast<const uint64_t*>(nearest), pass.npix,
        chain_cap, d_visible, pass.stats);
    FCU_LAUNCH("k_resolve_sunlit");
    k_fraction<<<(2 * frame.facets + 255) / 256, 256, 0, s>>>(2 * frame.facets, d_total, d_visible,
                                                              d_fraction);
    FCU_LAUNCH("k_fraction");
    FCU_CHECK(cudaMemcpyAsync(&stats, pass.stats, sizeof(RasterStats), cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaStreamSynchronize(s));
    refuse_fragments(stats);
}

}  // namespace facetcu
