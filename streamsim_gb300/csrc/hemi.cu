// hemi.cu — hemisphere ray-cast view factors and sun visibility over the LBVH.
//
// For every oriented side s (facet f = s / 2, normal N = +/- n_f) `rays` rays
// are cast: ray j of sample set (s mod sets) starts at a + u (b - a) + v (c - a)
// and leaves along T dx + Bt dy + N dz in the side's frame
// (T = normalize(helper x N), Bt = N x T).  A facet is hit when the
// Moller-Trumbore test accepts the ray at t > 0 and o + t d lies in the
// facet's box widened by the hit margin (the test's distance to a long thin
// facet met at a grazing angle can lie millimetres outside the facet; the
// BVH's leaf boxes are widened by twice the margin, so the traversal never
// culls a hit).  The nearest hit (smallest t, ties to the lower facet
// index, the origin facet skipped) gives the side seen: 2g if the ray
// meets g's normal side, 2g + 1 otherwise.  A warp per side then sorts the
// hit ids, counts runs, keeps the top_k most-hit sides (ties: lower side
// index) and writes the row sorted by neighbour with denominator = kept + sky
// rays.  With periodic tiles the nearest hit is taken over the scene and its
// copies (see Tiles).  Exactly the rules of the C oracle
// (orc_hemisphere_graph_periodic), so counts are comparable bit for bit: a
// row depends only on the set of its rays' hits, so the rays may be traced in
// any order.
//
// What the casting costs.  A ray of the 203,840-facet forest visits about 37
// four-wide nodes and tests 3 leaves (69 nodes in the binary tree); nothing
// comes from HBM, and the L1's passes (one per lane and load where lanes are
// at different nodes) and the ALU pipe bound it.  So nodes are 64 bytes, read
// with two loads (lbvh.cu), the rays of a block of facets are traced in the
// order of their directions, and lanes that are done take the next ray.  On
// that forest (208.7 M rays) the steps took: binary tree, a warp per side 156
// ms; cubic Morton cells 147; four-wide quantised nodes and a kernel of their
// own 110; sorted rays 95; refilled lanes 88 and with twice the L1 82;
// 32-byte loads 78 ms (2.7 G rays/s).
// This file is compiled with -fmad=false: the origin, direction and
// Moller-Trumbore arithmetic round like the oracle's.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <type_traits>

#include "internal.h"

namespace facetcu {
namespace {

constexpr int kWarps = 8;
constexpr uint32_t kSky = 0xFFFFFFFFu;
// A visited node leaves up to 3 children waiting, and the next one lies below it.
// Inner nodes below one another differ in the first bit that their leaves' keys
// don't share: 30 Morton bits, then those of the facet's place among equal codes,
// 30 for the 2^30 facets that setGeometry takes.
constexpr int kMortonBits = 30, kPlaceBits = 30;
constexpr int kStack = 180;
static_assert(kStack >= 3 * (kMortonBits + kPlaceBits), "no accepted scene overflows the stack");
constexpr int kKeptLeaves = 8;  // lanes with a leaf that make the warp test them (4, 12: equal; 16: +6 %)
constexpr int kRefill = 8;      // idle lanes that make the warp fetch rays (4, 12: equal)
constexpr int kSteps = 4;       // node steps between looks for idle lanes

struct Vec {
    float x, y, z;
};

__device__ __forceinline__ Vec vsub(Vec a, Vec b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ float vdot(Vec a, Vec b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ Vec vcross(Vec a, Vec b)
{
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ Vec pos(const facetcu_vertex& v)
{
    return {v.position[0], v.position[1], v.position[2]};
}

// Moller-Trumbore, the oracle's ray_triangle: t, or -1.
__device__ __forceinline__ float ray_triangle(Vec o, Vec d, Vec a, Vec e1, Vec e2)
{
    const Vec p = vcross(d, e2);
    const float det = vdot(e1, p);
    if (det == 0.0f) return -1.0f;
    const float inv = 1.0f / det;
    const Vec t0 = vsub(o, a);
    const float u = vdot(t0, p) * inv;
    if (u < 0.0f || u > 1.0f) return -1.0f;
    const Vec q = vcross(t0, e1);
    const float v = vdot(d, q) * inv;
    if (v < 0.0f || u + v > 1.0f) return -1.0f;
    const float t = vdot(e2, q) * inv;
    return t > 0.0f ? t : -1.0f;
}

// 1/d with |d| raised to at least 1e-24: the slab distances stay finite (no
// infinity, so no 0 * inf), and fminf/fmaxf order them.
__device__ __forceinline__ float safe_inv(float d)
{
    return 1.0f / (fabsf(d) < 1.0e-24f ? copysignf(1.0e-24f, d) : d);
}

// o + t d inside facet g's box widened by m (the hit rule's second half).
__device__ __forceinline__ bool in_hit_box(const facetcu_vertex* __restrict__ V, uint32_t g,
                                           Vec o, Vec d, float t, float m)
{
    const float p[3] = {o.x + t * d.x, o.y + t * d.y, o.z + t * d.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float v0 = V[3 * g].position[a], v1 = V[3 * g + 1].position[a],
                    v2 = V[3 * g + 2].position[a];
        const float lo = fminf(v0, fminf(v1, v2)) - m, hi = fmaxf(v0, fmaxf(v1, v2)) + m;
        if (!(p[a] >= lo && p[a] <= hi)) return false;
    }
    return true;
}

struct Hit {
    float t;
    uint32_t facet;
};

constexpr int kDone = INT_MIN;  // as kWideNone: no child, no more work

// One ray's way through the tree.  `cur` is the node it visits next, or kDone;
// `leaf` a leaf it has met and not tested yet (~index), or kDone.
struct Ray {
    Vec o, d, inv, noi;
    Hit best;
    int cur, leaf, sp;
    uint32_t skip;
};

__device__ __forceinline__ void start(Ray& r, Vec o, Vec d, uint32_t skip, uint32_t leaves)
{
    r.o = o;
    r.d = d;
    r.inv = {safe_inv(d.x), safe_inv(d.y), safe_inv(d.z)};
    r.noi = {-o.x * r.inv.x, -o.y * r.inv.y, -o.z * r.inv.z};
    r.sp = 0;
    r.skip = skip;
    r.leaf = leaves == 1 ? ~0 : kDone;
    r.cur = leaves == 1 ? kDone : 0;
}

// 32 bytes in one load: lanes at different nodes cost the L1 a pass per lane
// and load, whatever its width.
__device__ __forceinline__ void load32(const float4* p, float4& a, float4& b)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

__device__ __forceinline__ int pop(Ray& r, const int* stack) { return r.sp ? stack[--r.sp] : kDone; }

__device__ __forceinline__ float max3f(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// 1 + q / 128 of byte k (0x80 | q) of a word.
template <int K> __device__ __forceinline__ float plane(uint32_t w)
{
    return __uint_as_float(__byte_perm(w, 0x3F000000u, 0x7055 | (K << 8)));
}

// The four children of a node against the ray: a plane base + (1 + q / 128) S
// is met at v (S inv) + (base inv - o inv), one fma.  The roundings move a
// plane by about 1e-7 of the reach, a hundredth of the margin that the boxes
// carry beyond the hit rule's.  The nearest child is visited next, the others
// wait in the node's order: with 2-3 leaves tested per ray, sorting them all
// saves no visits (34.6 against 34.8 per ray on the forest).
__device__ __forceinline__ void node_step(Ray& r, const float4* __restrict__ nodes, int* stack,
                                          bool& overflow)
{
    const float4* n = nodes + 4 * size_t(r.cur);
    float4 A, B, C, D;
    load32(n, A, B);
    load32(n + 2, C, D);
    const float ax = A.w * r.inv.x, ay = B.x * r.inv.y, az = B.y * r.inv.z;
    const float cx = __fmaf_rn(A.x, r.inv.x, r.noi.x), cy = __fmaf_rn(A.y, r.inv.y, r.noi.y),
                cz = __fmaf_rn(A.z, r.inv.z, r.noi.z);
    const uint32_t lx = __float_as_uint(B.z), ly = __float_as_uint(B.w), lz = __float_as_uint(C.x),
                   hx = __float_as_uint(C.y), hy = __float_as_uint(C.z), hz = __float_as_uint(C.w);
    const bool px = r.inv.x > 0.0f, py = r.inv.y > 0.0f, pz = r.inv.z > 0.0f;
    const uint32_t nx = px ? lx : hx, fx = px ? hx : lx, ny = py ? ly : hy, fy = py ? hy : ly,
                   nz = pz ? lz : hz, fz = pz ? hz : lz;
    const int c[4] = {__float_as_int(D.x), __float_as_int(D.y), __float_as_int(D.z),
                      __float_as_int(D.w)};
    if (r.sp + 3 > kStack) {
        overflow = true;
        r.cur = kDone;
        return;
    }
    int next = kDone;
    auto test = [&](auto K) {
        constexpr int k = decltype(K)::value;
        const float tn = max3f(__fmaf_rn(plane<k>(nx), ax, cx), __fmaf_rn(plane<k>(ny), ay, cy),
                               fmaxf(__fmaf_rn(plane<k>(nz), az, cz), 0.0f));
        const float tf = min3f(__fmaf_rn(plane<k>(fx), ax, cx), __fmaf_rn(plane<k>(fy), ay, cy),
                               fminf(__fmaf_rn(plane<k>(fz), az, cz), r.best.t));
        const bool hit = tn <= tf, push = hit && next != kDone;
        if (push) stack[r.sp] = next;
        r.sp += push ? 1 : 0;
        next = hit ? c[k] : next;
    };
    test(std::integral_constant<int, 0>{});
    test(std::integral_constant<int, 1>{});
    test(std::integral_constant<int, 2>{});
    test(std::integral_constant<int, 3>{});
    if (next == kDone) next = pop(r, stack);
    r.cur = next;
}

__device__ __forceinline__ void leaf_step(Ray& r, const float4* __restrict__ tri,
                                          const facetcu_vertex* __restrict__ V, float m, bool any)
{
    const size_t k = 3 * size_t(~r.leaf);
    r.leaf = kDone;
    const float4 A = __ldg(tri + k), E1 = __ldg(tri + k + 1), E2 = __ldg(tri + k + 2);
    const uint32_t g = __float_as_uint(A.w);
    const float t = ray_triangle(r.o, r.d, {A.x, A.y, A.z}, {E1.x, E1.y, E1.z}, {E2.x, E2.y, E2.z});
    if (g != r.skip && t > 0.0f && (t < r.best.t || (t == r.best.t && g < r.best.facet)) &&
        in_hit_box(V, g, r.o, r.d, t, m)) {
        r.best.t = t;
        r.best.facet = g;
        if (any) r.cur = kDone;
    }
}

// Nearest hit (kAny = false) or occlusion (kAny = true) of the rays of a warp
// (lanes with `on`), improving on r.best.  Rays meet only a few leaves, so a
// lane keeps the leaf it meets and goes on; the warp tests the kept leaves
// once enough lanes hold one, or none can go on without.
template <bool kAny>
__device__ __forceinline__ bool trace(const float4* __restrict__ nodes,
                                      const float4* __restrict__ tri,
                                      const facetcu_vertex* __restrict__ V, float m, bool on, Ray& r)
{
    int stack[kStack];
    bool overflow = false;
    if (!on) r.cur = r.leaf = kDone;
    for (;;) {
#pragma unroll 1
        for (int k = 0; k < kSteps; ++k) {
            if (r.cur >= 0) node_step(r, nodes, stack, overflow);
            if (r.cur < 0 && r.cur != kDone && r.leaf == kDone) {
                r.leaf = r.cur;
                r.cur = pop(r, stack);
            }
        }
        const uint32_t kept = __ballot_sync(0xffffffffu, r.leaf != kDone);
        const uint32_t going = __ballot_sync(0xffffffffu, r.cur >= 0);
        if (__popc(kept) >= kKeptLeaves || !going) {
            if (!kept) break;
            if (r.leaf != kDone) leaf_step(r, tri, V, m, kAny);
        }
    }
    return !overflow;
}

struct Frame {
    Vec N, T, B;
};

// Periodic tiles (the raster mode's: the scene plus up to 20 copies offset by
// periodicTileOffset(t) x (periodicSizeX, periodicSizeZ)).  A copy is met by
// shifting the ray origin back by the tile's offset; the hit names the
// original facet; the origin facet is skipped in the scene's own tile only.
struct Tiles {
    float x[21], z[21];
    uint32_t n;
};

template <bool kAny>
__device__ __forceinline__ bool trace_tiles(const float4* __restrict__ nodes,
                                            const float4* __restrict__ tri,
                                            const facetcu_vertex* __restrict__ V, float m,
                                            uint32_t leaves, const Tiles& tiles, bool on, Vec o,
                                            Vec d, uint32_t skip, Hit& best)
{
    Ray r;
    r.best = {FLT_MAX, kSky};
    bool ok = true;
    for (uint32_t t = 0; t < tiles.n; ++t) {
        const bool more = on && !(kAny && r.best.facet != kSky);
        start(r, {o.x - tiles.x[t], o.y, o.z - tiles.z[t]}, d, t == 0 ? skip : kSky, leaves);
        ok &= trace<kAny>(nodes, tri, V, m, more, r);
    }
    best = r.best;
    return ok;
}

// The oracle's side_frame: helper = |N.y| < 0.9 ? +Y : +X.
__device__ __forceinline__ Frame side_frame(const facetcu_vertex* V, uint32_t s)
{
    const uint32_t f = s >> 1;
    Vec N = {V[3 * f].normal[0], V[3 * f].normal[1], V[3 * f].normal[2]};
    if (s & 1u) N = {-N.x, -N.y, -N.z};
    const Vec helper = fabsf(N.y) < 0.9f ? Vec{0.0f, 1.0f, 0.0f} : Vec{1.0f, 0.0f, 0.0f};
    const Vec t = vcross(helper, N);
    const float len = sqrtf(vdot(t, t));
    const float il = 1.0f / len;
    Frame fr;
    fr.N = N;
    fr.T = {t.x * il, t.y * il, t.z * il};
    fr.B = vcross(N, fr.T);
    return fr;
}

__device__ __forceinline__ Vec sample_origin(const facetcu_vertex* V, uint32_t f, float u, float v)
{
    const Vec a = pos(V[3 * f]);
    const Vec e1 = vsub(pos(V[3 * f + 1]), a);
    const Vec e2 = vsub(pos(V[3 * f + 2]), a);
    return {(a.x + e1.x * u) + e2.x * v, (a.y + e1.y * u) + e2.y * v, (a.z + e1.z * u) + e2.z * v};
}

// Sorts 32 E values of a warp, value lane * E + r in v[r] of the lane, by a
// bitonic network: exchanges nearer than E values apart stay in a lane's
// registers, the others are shuffles.  (The same network over shared memory
// took four times the instructions, most of them addresses and bank waits.)
template <int E>
__device__ __forceinline__ void warp_sort(uint32_t (&v)[E], int lane)
{
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j < E) {
#pragma unroll
                for (int r = 0; r < E; ++r) {
                    if (r & j) continue;
                    const bool up = k < E ? (r & k) == 0 : (lane & (k / E)) == 0;
                    const uint32_t lo = min(v[r], v[r | j]), hi = max(v[r], v[r | j]);
                    v[r] = up ? lo : hi;
                    v[r | j] = up ? hi : lo;
                }
            } else {
                const bool up = (lane & (k / E)) == 0, first = (lane & (j / E)) == 0;
#pragma unroll
                for (int r = 0; r < E; ++r) {
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], j / E);
                    v[r] = up == first ? min(v[r], o) : max(v[r], o);
                }
            }
        }
    }
}

// Warp-wide exclusive prefix sum of per-lane values.
__device__ __forceinline__ uint32_t warp_exclusive(uint32_t v, int lane, uint32_t& total)
{
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

// Rays a CTA sorts and traces: 2 CTAs of 512 threads and 54 KB leave half of
// the SM's memory to the L1 (32,768 rays: 8 % slower, 3 CTAs: 8 % slower, one
// CTA of 1,024 threads and 32,768 rays 3 % faster on the forest and 4 % slower
// on 4,096 facets).
constexpr uint32_t kBlockRays = 16384;
constexpr uint32_t kMaxBlockFacets = 64;
// Fewer facets per CTA where there would be fewer than 8 CTAs an SM, down to 768
// rays (setting up and sorting a CTA costs as much as tracing some hundred), or one
// CTA an SM.  The whole graph in us with a warp per side / 8 CTAs an SM and no
// least number / so / 1,024 rays at least:
//     1,936 facets  32 rays   172   238   173   176
//                  100 rays   453   352   279   271
//     2,916 facets  32 rays   186         188   194
//     4,096 facets  32 rays   334   276   227   204
//                   64 rays   415   356   302   286
//    10,800 facets  48 rays   946   601   593   595
constexpr uint32_t kBlocksPerSm = 8, kLeastRays = 768;
constexpr uint32_t kBins = 4096;      // directions: 64 x 64 cells of the octahedral map
constexpr int kTraceThreads = 512;

__device__ __forceinline__ uint32_t spread6(uint32_t v)
{
    v = (v | (v << 4)) & 0x30Fu;
    v = (v | (v << 2)) & 0x333u;
    return (v | (v << 1)) & 0x555u;
}
// Cell of a direction: Morton number in the octahedral map of the sphere.
__device__ __forceinline__ uint32_t direction_cell(Vec d)
{
    const float inv = 1.0f / (fabsf(d.x) + fabsf(d.y) + fabsf(d.z));
    float u = d.x * inv, v = d.z * inv;
    if (d.y < 0.0f) {
        const float a = (1.0f - fabsf(v)) * copysignf(1.0f, u);
        v = (1.0f - fabsf(u)) * copysignf(1.0f, v);
        u = a;
    }
    const uint32_t iu = min(uint32_t(fmaxf((u + 1.0f) * 32.0f, 0.0f)), 63u);
    const uint32_t iv = min(uint32_t(fmaxf((v + 1.0f) * 32.0f, 0.0f)), 63u);
    return spread6(iu) | (spread6(iv) << 1);
}

// Hit ids of the rays of facets [first, last) in tree order, both sides:
// hits[2 (k - first) + side][ray].  A CTA takes `per_block` neighbouring facets
// and sorts their rays by direction, so that a warp's rays run side by side
// (the rays of one side leave one point in all directions): 22 of 32 lanes
// are busy, with 16 for rays in a side's own order.
__global__ void __launch_bounds__(kTraceThreads, 2) k_hemi_trace(
    const facetcu_vertex* __restrict__ V, const float4* __restrict__ nodes,
    const float4* __restrict__ tri, uint32_t leaves, uint32_t first, uint32_t last,
    uint32_t per_block, const float* __restrict__ uv, const float* __restrict__ dirs, uint32_t rays,
    uint32_t sets, uint32_t shift, Tiles tiles, float hit_m, uint32_t* hits, uint32_t* error)
{
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t bin[kBins];
    __shared__ float frames[2 * kMaxBlockFacets][9];
    __shared__ uint32_t facet[kMaxBlockFacets];
    __shared__ uint32_t warp_sum[kTraceThreads / 32], total, next;
    uint16_t* order = reinterpret_cast<uint16_t*>(smem);
    const uint32_t k0 = first + blockIdx.x * per_block, n = min(per_block, last - k0);
    const uint32_t sides = 2 * n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < kBins; i += kTraceThreads) bin[i] = 0;
    if (threadIdx.x < n) facet[threadIdx.x] = __float_as_uint(tri[3 * size_t(k0 + threadIdx.x)].w);
    __syncthreads();
    if (threadIdx.x < sides) {
        const Frame fr = side_frame(V, 2 * facet[threadIdx.x >> 1] + (threadIdx.x & 1));
        float* q = frames[threadIdx.x];
        q[0] = fr.T.x; q[1] = fr.T.y; q[2] = fr.T.z;
        q[3] = fr.B.x; q[4] = fr.B.y; q[5] = fr.B.z;
        q[6] = fr.N.x; q[7] = fr.N.y; q[8] = fr.N.z;
    }
    if (threadIdx.x == 0) next = 0;
    __syncthreads();
    auto direction = [&](uint32_t ls, uint32_t j) {
        const uint32_t s = 2 * facet[ls >> 1] + (ls & 1);
        const size_t k = size_t(s % sets) * rays + j;
        const float dx = dirs[3 * k], dy = dirs[3 * k + 1], dz = dirs[3 * k + 2];
        const float* q = frames[ls];
        return Vec{q[0] * dx + q[3] * dy + q[6] * dz, q[1] * dx + q[4] * dy + q[7] * dz,
                   q[2] * dx + q[5] * dy + q[8] * dz};
    };
    for (uint32_t i = threadIdx.x; i < sides << shift; i += kTraceThreads) {
        const uint32_t j = i & ((1u << shift) - 1u);
        if (j < rays) atomicAdd(&bin[direction_cell(direction(i >> shift, j))], 1u);
    }
    __syncthreads();
    {   // exclusive scan of the bins
        constexpr uint32_t kPer = kBins / kTraceThreads;
        uint32_t v[kPer], sum = 0;
        for (uint32_t k = 0; k < kPer; ++k) {
            v[k] = bin[threadIdx.x * kPer + k];
            sum += v[k];
        }
        uint32_t t;
        uint32_t at = warp_exclusive(sum, int(lane), t);
        if (lane == 0) warp_sum[warp] = t;
        __syncthreads();
        for (uint32_t w = 0; w < warp; ++w) at += warp_sum[w];
        for (uint32_t k = 0; k < kPer; ++k) {
            bin[threadIdx.x * kPer + k] = at;
            at += v[k];
        }
        if (threadIdx.x == kTraceThreads - 1) total = at;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < sides << shift; i += kTraceThreads) {
        const uint32_t j = i & ((1u << shift) - 1u);
        if (j < rays) order[atomicAdd(&bin[direction_cell(direction(i >> shift, j))], 1u)] = uint16_t(i);
    }
    __syncthreads();
    const uint32_t count = total;
    int stack[kStack];
    bool overflow = false, busy = false, more = true;
    uint32_t i = 0, tile = 0;
    Ray r;
    r.cur = r.leaf = kDone;
    for (;;) {
        if (busy && r.cur == kDone && r.leaf == kDone) {  // this copy of the scene is done
            const uint32_t ls = i >> shift, j = i & ((1u << shift) - 1u);
            if (++tile < tiles.n && !overflow) {
                const uint32_t f = facet[ls >> 1], s = 2 * f + (ls & 1);
                const size_t k = size_t(s % sets) * rays + j;
                const Vec o = sample_origin(V, f, uv[2 * k], uv[2 * k + 1]);
                start(r, {o.x - tiles.x[tile], o.y, o.z - tiles.z[tile]}, r.d, kSky, leaves);
            } else {
                uint32_t id = kSky;
                const uint32_t g = r.best.facet;
                if (g != kSky) {
                    const Vec ng = {V[3 * g].normal[0], V[3 * g].normal[1], V[3 * g].normal[2]};
                    id = 2u * g + (vdot(ng, r.d) < 0.0f ? 0u : 1u);
                }
                hits[(size_t(2) * (k0 - first) + ls) * rays + j] = id;
                busy = false;
            }
        }
        const uint32_t idle = __ballot_sync(0xffffffffu, !busy);
        if (more && __popc(idle) >= kRefill) {
            uint32_t r0 = 0;
            if (lane == 0) r0 = atomicAdd(&next, uint32_t(__popc(idle)));
            r0 = __shfl_sync(0xffffffffu, r0, 0);
            more = r0 + __popc(idle) < count;
            const uint32_t at = r0 + __popc(idle & ((1u << lane) - 1u));
            if (!busy && at < count) {
                i = order[at];
                const uint32_t ls = i >> shift, j = i & ((1u << shift) - 1u);
                const uint32_t f = facet[ls >> 1], s = 2 * f + (ls & 1);
                const size_t k = size_t(s % sets) * rays + j;
                const Vec d = direction(ls, j);
                start(r, sample_origin(V, f, uv[2 * k], uv[2 * k + 1]), d, f, leaves);
                r.best = {FLT_MAX, kSky};
                tile = 0;
                busy = true;
            }
        } else if (idle == 0xffffffffu) {
            break;
        }
#pragma unroll 1
        for (int n = 0; n < kSteps; ++n) {
            if (r.cur >= 0) node_step(r, nodes, stack, overflow);
            if (r.cur < 0 && r.cur != kDone && r.leaf == kDone) {
                r.leaf = r.cur;
                r.cur = pop(r, stack);
            }
            const uint32_t kept = __ballot_sync(0xffffffffu, r.leaf != kDone);
            const uint32_t going = __ballot_sync(0xffffffffu, r.cur >= 0);
            if (__popc(kept) >= kKeptLeaves || !going) {
                if (!kept) break;
                if (r.leaf != kDone) leaf_step(r, tri, V, hit_m, false);
            }
        }
    }
    if (overflow) atomicExch(error, 1u);
}

// A side's row from its rays' hit ids, a warp per side (E values per lane):
// sorted ids, the runs' lengths as counts, the top_k most-hit sides (ties: the
// lower side) in side order.
template <int E>
__global__ void __launch_bounds__(kWarps * 32) k_hemi_rows(
    const float4* __restrict__ tri, uint32_t first, uint32_t last,
    const uint32_t* __restrict__ traced, uint32_t rays, uint32_t top_k, uint2* __restrict__ edges,
    uint32_t* nnz, uint32_t* denom, uint32_t* skyc, unsigned long long* dropped)
{
    __shared__ uint32_t ids[kWarps][32 * E];
    __shared__ uint16_t starts[kWarps][32 * E + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* uniq = ids[warp];
    uint16_t* start = starts[warp];
    const uint32_t row = blockIdx.x * kWarps + warp;
    if (row >= 2 * (last - first)) return;  // (whole warps)
    const uint32_t s = 2 * __float_as_uint(tri[3 * size_t(first + (row >> 1))].w) + (row & 1);
    uint32_t v[E];
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const uint32_t j = uint32_t(r) * 32 + lane;
        v[r] = j < rays ? __ldcs(traced + size_t(row) * rays + j) : kSky;
    }
    warp_sort<E>(v, lane);
    uint32_t before = __shfl_up_sync(0xffffffffu, v[E - 1], 1);
    if (lane == 0) before = kSky;
    uint32_t heads = 0, found = 0;
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const uint32_t prev = r ? v[r > 0 ? r - 1 : 0] : before;
        found += v[r] != kSky ? 1u : 0u;
        heads += v[r] != kSky && v[r] != prev ? 1u : 0u;
    }
    uint32_t unique;
    uint32_t at = warp_exclusive(heads, lane, unique);
    const uint32_t nonsky = __reduce_add_sync(0xffffffffu, found);
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const uint32_t prev = r ? v[r > 0 ? r - 1 : 0] : before;
        if (v[r] != kSky && v[r] != prev) {
            uniq[at] = v[r];
            start[at] = uint16_t(lane * E + r);
            ++at;
        }
    }
    if (lane == 0) start[unique] = uint16_t(nonsky);
    __syncwarp();
    auto count = [&](uint32_t i) { return uint32_t(start[i + 1]) - uint32_t(start[i]); };
    uint2* out = edges + size_t(s) * top_k;
    uint32_t keep = unique, kept = nonsky;
    if (unique <= top_k) {
        for (uint32_t i = lane; i < unique; i += 32) out[i] = make_uint2(uniq[i], count(i));
    } else {
        // keep every count above T, and in side order the first ones equal to
        // T, where T is the least with no more than top_k above it
        keep = top_k;
        uint32_t T = 0, above = unique;
        while (above > top_k) {
            ++T;
            uint32_t n = 0;
            for (uint32_t i = lane; i < unique; i += 32) n += count(i) > T ? 1u : 0u;
            above = __reduce_add_sync(0xffffffffu, n);
        }
        uint32_t equal_left = top_k - above, w = 0;
        kept = 0;
        const uint32_t below = (1u << lane) - 1u;
        for (uint32_t i0 = 0; i0 < unique; i0 += 32) {
            const uint32_t i = i0 + lane;
            const uint32_t c = i < unique ? count(i) : 0u;
            const uint32_t eq = __ballot_sync(0xffffffffu, i < unique && c == T);
            const bool take = i < unique && (c > T || (c == T && uint32_t(__popc(eq & below)) < equal_left));
            const uint32_t taken = __ballot_sync(0xffffffffu, take);
            if (take) {
                out[w + __popc(taken & below)] = make_uint2(uniq[i], c);
                kept += c;
            }
            w += __popc(taken);
            equal_left -= min(equal_left, uint32_t(__popc(eq)));
        }
        kept = __reduce_add_sync(0xffffffffu, kept);
    }
    if (lane == 0) {
        const uint32_t sky = rays - nonsky;
        nnz[s] = keep;
        skyc[s] = sky;
        denom[s] = kept + sky;
        if (kept < nonsky) atomicAdd(dropped, (unsigned long long)(nonsky - kept));
    }
}

__global__ void k_hemi_compact(const uint2* __restrict__ tmp, const uint32_t* __restrict__ rows,
                               uint32_t surfaces, uint32_t top_k, uint2* __restrict__ edges)
{
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= surfaces) return;
    const uint32_t b = rows[warp], n = rows[warp + 1] - b;
    for (uint32_t i = lane; i < n; i += 32) edges[b + i] = __ldcs(tmp + size_t(warp) * top_k + i);
}

__global__ void k_set_total(uint32_t* rows, uint32_t n, const unsigned long long* total)
{
    rows[n] = uint32_t(*total);
}

// Occlusion toward the sun from `samples` points of the side facing it (at
// most one of a facet's does), `share` neighbouring warps per facet.
__global__ void __launch_bounds__(256) k_hemi_sunlit(const facetcu_vertex* __restrict__ V,
                                                     const float4* __restrict__ nodes,
                                                     const float4* __restrict__ tri, uint32_t leaves,
                                                     uint32_t surfaces, const float* __restrict__ uv,
                                                     uint32_t samples, uint32_t sets, Vec sun,
                                                     Tiles tiles, float hit_m, uint32_t share,
                                                     float* fraction, uint32_t* error)
{
    __shared__ uint32_t part_lit[8];
    const uint32_t warp = threadIdx.x >> 5, part = warp % share;
    const uint32_t f = (blockIdx.x * 8 + warp) / share;
    const int lane = threadIdx.x & 31;
    if (share == 1 && 2 * f >= surfaces) return;
    const bool valid = 2 * f < surfaces;
    uint32_t lit = 0, s = 0;
    bool up = false, down = false;
    if (valid) {
        const Vec n = {V[3 * f].normal[0], V[3 * f].normal[1], V[3 * f].normal[2]};
        const Vec back = {-n.x, -n.y, -n.z};
        up = vdot(n, sun) > 0.0f;
        down = vdot(back, sun) > 0.0f;
        if (part == 0 && lane < 2 && !(lane ? down : up)) fraction[2 * f + lane] = 0.0f;
        s = 2 * f + (up ? 0u : 1u);
    }
    if (up || down) {
        const uint32_t set = s % sets;
        for (uint32_t j0 = part * 32; j0 < samples; j0 += 32 * share) {
            const uint32_t j = j0 + lane;
            const bool on = j < samples;
            const size_t k = size_t(set) * samples + (on ? j : 0);
            const Vec o = sample_origin(V, f, uv[2 * k], uv[2 * k + 1]);
            Hit h;
            if (!trace_tiles<true>(nodes, tri, V, hit_m, leaves, tiles, on, o, sun, f, h))
                atomicExch(error, 1u);
            if (on && h.facet == kSky) ++lit;
        }
        lit = __reduce_add_sync(0xffffffffu, lit);
    }
    if (share > 1) {
        if (lane == 0) part_lit[warp] = lit;
        __syncthreads();
        if (part) return;
        for (uint32_t k = 1; k < share; ++k) lit += part_lit[warp + k];
    }
    if (lane == 0 && (up || down)) fraction[s] = float(lit) / float(samples);
}

Tiles make_tiles(const PeriodicTiles& p)
{
    Tiles t{};
    t.n = std::min<uint32_t>(p.count, 20u) + 1u;
    for (uint32_t i = 0; i < t.n; ++i) {
        t.x[i] = p.dx[i];
        t.z[i] = p.dz[i];
    }
    return t;
}

}  // namespace

void hemisphere_graph(const facetcu_vertex* d_vertices, uint32_t facets, const Lbvh& bvh,
                      const float* d_uv, const float* d_dir, uint32_t rays, uint32_t sets,
                      uint32_t top_k, const PeriodicTiles& periodic, DeviceGraph& g,
                      unsigned long long* dropped, Workspace& ws, cudaStream_t s)
{
    const uint32_t S = 2u * facets;
    top_k = std::min(top_k, rays);
    g.surfaces = S;
    ScratchBuffer tmp(ws), counters(ws);
    uint2* tmp_edges = static_cast<uint2*>(tmp.reserve(size_t(S) * top_k * 8 + 8));
    uint32_t* rows = static_cast<uint32_t*>(g.row_offsets.reserve((size_t(S) + 1) * 4));
    uint32_t* den = static_cast<uint32_t*>(g.denominators.reserve(size_t(S) * 4));
    uint32_t* sky = static_cast<uint32_t*>(g.sky.reserve(size_t(S) * 4));
    char* cnt = static_cast<char*>(counters.reserve(64));
    unsigned long long* d_dropped = reinterpret_cast<unsigned long long*>(cnt);
    unsigned long long* d_total = reinterpret_cast<unsigned long long*>(cnt + 8);
    uint32_t* d_error = reinterpret_cast<uint32_t*>(cnt + 16);
    FCU_CHECK(cudaMemsetAsync(cnt, 0, 64, s));
    uint32_t shift = 5;
    while ((1u << shift) < rays) ++shift;
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    sms = std::max(sms, 1);
    const uint32_t even = std::max(facets / (kBlocksPerSm * uint32_t(sms)),
                                   std::min(kLeastRays >> (shift + 1), facets / uint32_t(sms)));
    const uint32_t per_block =
        std::max(1u, std::min({kMaxBlockFacets, kBlockRays >> (shift + 1), even}));
    // hit ids of a run of facets at a time
    const uint32_t run = std::min(facets, std::max(per_block, uint32_t((size_t(1) << 30) / (size_t(8) * rays)) / per_block * per_block));
    ScratchBuffer traced_buf(ws);
    uint32_t* traced = static_cast<uint32_t*>(traced_buf.reserve(size_t(run) * 2 * rays * 4));
    const size_t smem_trace = size_t(2) * (size_t(2) * per_block << shift);
    // (the limit belongs to the function, not to this context: always the most)
    FCU_CHECK(cudaFuncSetAttribute(k_hemi_trace, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(2 * kBlockRays)));
    for (uint32_t f0 = 0; f0 < facets; f0 += run) {
        const uint32_t f1 = std::min(facets, f0 + run);
        k_hemi_trace<<<(f1 - f0 + per_block - 1) / per_block, kTraceThreads, smem_trace, s>>>(
            d_vertices, bvh.nodes.as<float4>(), bvh.tri.as<float4>(), bvh.leaves, f0, f1, per_block,
            d_uv, d_dir, rays, sets, shift, make_tiles(periodic), bvh.hit_margin, traced, d_error);
        FCU_LAUNCH("k_hemi_trace");
        auto make_rows = [&](auto kernel) {
            kernel<<<(2 * (f1 - f0) + kWarps - 1) / kWarps, kWarps * 32, 0, s>>>(
                bvh.tri.as<float4>(), f0, f1, traced, rays, top_k, tmp_edges, rows, den, sky,
                d_dropped);
        };
        switch (shift) {
        case 5: make_rows(k_hemi_rows<1>); break;
        case 6: make_rows(k_hemi_rows<2>); break;
        case 7: make_rows(k_hemi_rows<4>); break;
        case 8: make_rows(k_hemi_rows<8>); break;
        case 9: make_rows(k_hemi_rows<16>); break;
        default: make_rows(k_hemi_rows<32>); break;  // rays <= 1023
        }
        FCU_LAUNCH("k_hemi_rows");
    }
    // rows currently holds per-side nnz; scan in place into offsets
    exclusive_scan_u32(rows, rows, S, d_total, ws, s);
    k_set_total<<<1, 1, 0, s>>>(rows, S, d_total);
    FCU_LAUNCH("k_set_total");
    unsigned long long host[3] = {0, 0, 0};
    FCU_CHECK(cudaMemcpyAsync(host, cnt, 24, cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaStreamSynchronize(s));
    if (uint32_t(host[2])) throw Error(FACETCU_DEVICE_CAPACITY, "BVH traversal stack exceeded 180 entries");
    g.nnz = host[1];
    facetcu_csr_edge* edges = static_cast<facetcu_csr_edge*>(g.edges.reserve((g.nnz + 1) * 8));
    k_hemi_compact<<<(S * 32 + 255) / 256, 256, 0, s>>>(tmp_edges, rows, S, top_k, reinterpret_cast<uint2*>(edges));
    FCU_LAUNCH("k_hemi_compact");
    FCU_CHECK(cudaStreamSynchronize(s));
    g.changed();
    if (dropped) *dropped = host[0];
}

void hemisphere_sunlit(const facetcu_vertex* d_vertices, uint32_t facets, const Lbvh& bvh,
                       const float* d_uv, uint32_t samples, uint32_t sets, float3 sun,
                       const PeriodicTiles& periodic, float* d_fraction, Workspace& ws,
                       cudaStream_t s)
{
    const uint32_t S = 2u * facets;
    ScratchBuffer err(ws);
    uint32_t* d_error = static_cast<uint32_t*>(err.reserve(16));
    FCU_CHECK(cudaMemsetAsync(d_error, 0, 16, s));
    // Several warps to a facet where there are fewer facets than warps to run
    // (64 an SM; twice as many share the rays of uneven facets better): 256
    // samples of 4,096 facets 160 us with one, 137, 131 and 124 from 32, 64 and
    // 128 warps an SM.
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    uint32_t share = 1;
    while (share < 8 && share * 32 < samples && facets * share < uint32_t(sms) * 128u) share *= 2;
    k_hemi_sunlit<<<unsigned((uint64_t(facets) * share + 7) / 8), 256, 0, s>>>(
        d_vertices, bvh.nodes.as<float4>(), bvh.tri.as<float4>(), bvh.leaves, S, d_uv, samples, sets,
        {sun.x, sun.y, sun.z}, make_tiles(periodic), bvh.hit_margin, share, d_fraction, d_error);
    FCU_LAUNCH("k_hemi_sunlit");
    uint32_t e = 0;
    FCU_CHECK(cudaMemcpyAsync(&e, d_error, 4, cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaStreamSynchronize(s));
    if (e) throw Error(FACETCU_DEVICE_CAPACITY, "BVH traversal stack exceeded 180 entries");
}

}  // namespace facetcu
