// column.cu — sweeps of ONE right-hand side over a large graph, with the
// neighbour values gathered from shared memory.
//
// A one-column sweep reads one 4-byte value per edge.  From L2 that costs a
// 32-byte sector each (75 M edges x 32 B = 2.4 GB per sweep on the
// 200,000-facet forest) and the L1's one tag look-up per lane, so the gather,
// not the edge list, bounds it.  Here the column is cut into tiles of kTile
// sides that fill a shared memory.  A CTA (one per SM) holds one tile and
// streams the edges of a range of rows into it, a share of the tile's edges
// set by their number; the sum of a (row, tile) pair goes to a partial array
// [tile][side], and a second kernel adds a side's partials in tile order and
// forms the new value.  HBM sees the edge words once; the partials (4 bytes
// per tile and side) stay in L2.  The order of all additions is fixed.
//
// The edge words of a tile are laid out for that loop: within a window of
// kWindow rows, rows sorted by their number of edges in the tile, 32 rows to
// a group, the words of a group interleaved (word k of all 32 rows, then word
// k + 1), so that a lane owns a row and the warp reads 128 consecutive bytes.
// The plan is made on the device once per graph.
//
// (The other split, a CTA per row range that walks all tiles and keeps the
// row sums itself, reads the whole column in every CTA and meets a barrier
// per tile: 289 us per sweep on a 200,000-facet, 84 M-edge exchange graph,
// against 87 here and 340 for one thread per facet over the CSR.)
#include <algorithm>
#include <cmath>
#include <vector>

#include "compensated.cuh"
#include "internal.h"
#include "sweep_math.cuh"

namespace facetcu {
namespace {

constexpr uint32_t kTile = 49152;    // sides per tile (192 KB)
constexpr uint32_t kMaxTiles = 16;   // (tile, row) tables while the plan is made; partials
constexpr uint32_t kWindow = 4096;   // rows sorted together
constexpr uint32_t kWinBits = 12;
// A word: the side within the tile in the low 16 bits, the count as a BF16
// number in the high ones, so that masking turns it into the float factor.  A
// count with more than 8 significant bits takes two words (its high and its
// low byte).  A word of count 0 at side kTile, where the tile holds a zero,
// fills up the shorter rows of a group.
constexpr uint32_t kPad = kTile;
constexpr uint32_t kMaxCount = 0xffffu;
constexpr uint32_t kGroupCost = 4;   // of a group beside its words, in words, when work is split
constexpr int kThreads = 1024;
// Fewer edges: the fixed cost of a sweep (tiles, two launches: 14 us) takes what
// the gather saves.  From here on one column of the batched solver, the making of
// the plan included, is faster than over the CSR, whose renumbered copy it does
// not need (first call, 9 sweeps: 15.9 M edges 1.37 ms against 1.82, 83.8 M 3.6
// against 6.6).
constexpr uint64_t kMinEdges = 10u << 20;
// Mean edges of a (row, tile) pair: with 3.5 (13 M edges, 400,000 sides) 33 us
// a sweep against 49; fewer leave more group heads and partials than edges.
constexpr uint64_t kMinTileEdges = 3;
static_assert(kTile < 0xffffu && kTile % 4 == 0 && kWindow == 1u << kWinBits, "fields");

struct Share {  // of a CTA: its tile, and the tile's groups [begin, end)
    uint32_t tile, begin, end;
};
struct View {
    const Share* shares;
    const uint2* groups;   // first word / 32, first row of the window
    const uint32_t* meta;  // [group][32] row within the window | edges << 16
    const uint32_t* words;
    uint32_t tiles, surfaces;
};

inline unsigned blocks(size_t n, unsigned b) { return unsigned((n + b - 1) / b); }

// ---- the plan ------------------------------------------------------------
__device__ __forceinline__ void edge(const uint32_t* packed, const facetcu_csr_edge* edges,
                                     uint32_t nb_bits, size_t e, uint32_t& nb, uint32_t& c)
{
    if (packed) {
        const uint32_t p = __ldg(packed + e);
        nb = p & ((1u << nb_bits) - 1u);
        c = p >> nb_bits;
    } else {
        nb = edges[e].neighbor;
        c = edges[e].count;
    }
}

// The words of a count: its BF16 parts (the second is 0 for most).
__device__ __forceinline__ uint2 parts_of(uint32_t count)
{
    const float f = float(count);  // exact: at most 16 bits
    const uint32_t bits = __float_as_uint(f);
    if ((bits & 0xffffu) == 0u) return make_uint2(bits, 0u);
    return make_uint2(__float_as_uint(float(count & 0xff00u)), __float_as_uint(float(count & 0xffu)));
}

// Words of every row in every tile, a warp per row; seg is [tile][row].
__global__ void __launch_bounds__(256) k_count(const uint32_t* rows, const uint32_t* packed,
                                               const facetcu_csr_edge* edges, uint32_t nb_bits,
                                               uint32_t S, uint32_t tiles, uint16_t* seg,
                                               uint32_t* longest)
{
    __shared__ uint32_t cnt[8][kMaxTiles];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t r = blockIdx.x * 8 + warp;
    if (r >= S) return;
    if (lane < tiles) cnt[warp][lane] = 0;
    __syncwarp();
    const uint32_t end = rows[r + 1];
    for (uint32_t e = rows[r] + lane; e < end; e += 32) {
        uint32_t nb, c;
        edge(packed, edges, nb_bits, e, nb, c);
        atomicAdd(&cnt[warp][nb / kTile], parts_of(c).y ? 2u : 1u);
    }
    __syncwarp();
    if (lane < tiles) {
        const uint32_t c = cnt[warp][lane];
        seg[size_t(lane) * S + r] = uint16_t(c);
        if (c > 0xffffu) atomicMax(longest, c);
    }
}

// Groups of every (tile, window): its rows with edges, 32 at a time.
__global__ void __launch_bounds__(256) k_groups(uint32_t S, uint32_t windows, const uint16_t* seg,
                                                uint32_t* ngroups)
{
    const uint32_t t = blockIdx.x / windows, w = blockIdx.x % windows;
    const uint32_t r0 = w * kWindow, n = min(kWindow, S - r0);
    uint32_t k = 0;
    for (uint32_t i = threadIdx.x; i < n; i += 256) k += seg[size_t(t) * S + r0 + i] != 0;
    __shared__ uint32_t sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    k = __reduce_add_sync(0xffffffffu, k);
    if ((threadIdx.x & 31) == 0) atomicAdd(&sum, k);
    __syncthreads();
    if (threadIdx.x == 0) ngroups[blockIdx.x] = (sum + 31) / 32;
}

// Slots of one (tile, window): rows with edges, longest first.
__global__ void __launch_bounds__(256) k_order(uint32_t S, uint32_t windows, const uint16_t* seg,
                                               const uint32_t* first_group, uint16_t* slot,
                                               uint32_t* meta, uint32_t* glen)
{
    constexpr uint32_t kBins = 1024;  // longer rows share the last bin
    __shared__ uint32_t hist[kBins];
    __shared__ uint32_t len_of[kWindow / 32];
    __shared__ uint32_t warp_sum[8], used;
    const uint32_t t = blockIdx.x / windows, w = blockIdx.x % windows;
    const uint32_t r0 = w * kWindow, n = min(kWindow, S - r0);
    const size_t g0 = first_group[blockIdx.x], c0 = size_t(t) * S + r0;
    for (uint32_t i = threadIdx.x; i < kBins; i += 256) hist[i] = 0;
    if (threadIdx.x < kWindow / 32) len_of[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += 256) {
        const uint32_t l = seg[c0 + i];
        if (l) atomicAdd(&hist[min(l, kBins - 1)], 1u);
    }
    __syncthreads();
    // start of each bin, longest bins first: thread i owns bins
    // kBins - 1 - 4 i - {0..3}
    uint32_t b[4], sum = 0;
    for (int k = 0; k < 4; ++k) {
        b[k] = hist[kBins - 1 - (threadIdx.x * 4 + k)];
        sum += b[k];
    }
    uint32_t incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((threadIdx.x & 31) >= uint32_t(o)) incl += y;
    }
    if ((threadIdx.x & 31) == 31) warp_sum[threadIdx.x >> 5] = incl;
    __syncthreads();
    uint32_t before = incl - sum;
    for (uint32_t k = 0; k < (threadIdx.x >> 5); ++k) before += warp_sum[k];
    if (threadIdx.x == 255) used = before + sum;
    for (int k = 0; k < 4; ++k) {
        hist[kBins - 1 - (threadIdx.x * 4 + k)] = before;
        before += b[k];
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += 256) {
        const uint32_t l = seg[c0 + i];
        if (!l) continue;
        const uint32_t k = atomicAdd(&hist[min(l, kBins - 1)], 1u);
        slot[c0 + i] = uint16_t(k);
        meta[(g0 + (k >> 5)) * 32 + (k & 31)] = i | (l << 16);
        atomicMax(&len_of[k >> 5], l);
    }
    __syncthreads();
    const uint32_t ng = (used + 31) / 32;
    for (uint32_t k = used + threadIdx.x; k < ng * 32; k += 256)
        meta[(g0 + (k >> 5)) * 32 + (k & 31)] = 0;  // no row
    if (threadIdx.x < ng) glen[g0 + threadIdx.x] = len_of[threadIdx.x];
}

// Share k of n of a tile's groups, by words and groups.
__global__ void k_split(const uint32_t* woff, uint32_t slots, uint32_t total, const Share* shares,
                        const uint32_t* tile_group, uint32_t ctas, Share* out)
{
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ctas) return;
    const Share sh = shares[p];  // tile, share k, shares n
    const uint32_t g0 = tile_group[sh.tile], g1 = tile_group[sh.tile + 1];
    auto cost = [&](uint32_t g) {
        return uint64_t((g < slots ? woff[g] : total) - woff[g0]) + uint64_t(kGroupCost) * (g - g0);
    };
    auto at = [&](uint32_t k) {
        const uint64_t want = cost(g1) * k / sh.end;
        uint32_t lo = g0, hi = g1;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (cost(mid) < want) lo = mid + 1;
            else hi = mid;
        }
        return k >= sh.end ? g1 : lo;
    };
    out[p] = {sh.tile, at(sh.begin), at(sh.begin + 1)};
}

// {first word / 32, first row} of every group.
__global__ void __launch_bounds__(128) k_group_info(uint32_t windows, const uint32_t* first_group,
                                                    const uint32_t* ngroups, const uint32_t* woff,
                                                    uint2* groups)
{
    const uint32_t g0 = first_group[blockIdx.x];
    if (threadIdx.x < ngroups[blockIdx.x])
        groups[g0 + threadIdx.x] =
            make_uint2(woff[g0 + threadIdx.x], (blockIdx.x % windows) * kWindow);
}

__global__ void k_fill(uint4* words, size_t n)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) words[i] = make_uint4(kPad, kPad, kPad, kPad);
}

// Every edge to its word, a warp per row; a row's edges keep their order, the
// low bytes of the rare large counts come last.
__global__ void __launch_bounds__(256) k_scatter(const uint32_t* rows, const uint32_t* packed,
                                                 const facetcu_csr_edge* edges, uint32_t nb_bits,
                                                 uint32_t S, uint32_t tiles, uint32_t windows,
                                                 const uint32_t* first_group, const uint16_t* slot,
                                                 const uint32_t* woff, uint32_t* words)
{
    __shared__ uint32_t cnt[8][kMaxTiles];
    __shared__ size_t base[8][kMaxTiles];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t r = blockIdx.x * 8 + warp;
    if (r >= S) return;
    const uint32_t begin = rows[r], end = rows[r + 1];
    if (begin == end) return;
    if (lane < tiles) {
        cnt[warp][lane] = 0;
        // (a pair without edges has no slot: its base is not used)
        const uint32_t sl = slot[size_t(lane) * S + r];
        const uint32_t g = first_group[lane * windows + (r >> kWinBits)] + (sl >> 5);
        base[warp][lane] = size_t(woff[g]) * 32 + (sl & 31);
    }
    __syncwarp();
    bool second = false;
    for (int pass = 0; pass < 2; ++pass) {
        for (uint32_t e0 = begin; e0 < end; e0 += 32) {
            const uint32_t e = e0 + lane;
            uint32_t nb = 0, c = 0;
            if (e < end) edge(packed, edges, nb_bits, e, nb, c);
            const uint2 parts = parts_of(c);
            second |= parts.y != 0u;
            const bool on = e < end && (pass == 0 || parts.y);
            const uint32_t t = on ? nb / kTile : 0xffffffffu;
            const uint32_t peers = __match_any_sync(0xffffffffu, t);
            const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
            if (on)
                words[base[warp][t] + size_t(cnt[warp][t] + rank) * 32] =
                    (nb - t * kTile) | (pass == 0 ? parts.x : parts.y);
            __syncwarp();
            if (on && rank == 0) cnt[warp][t] += __popc(peers);
            __syncwarp();
        }
        if (!__any_sync(0xffffffffu, second)) break;
    }
}

// ---- the sweep -------------------------------------------------------------
__device__ __forceinline__ void cp_async16(float* dst, const float* src)
{
    const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Compensated accumulation (TwoProduct and Neumaier's TwoSum): sum + c holds
// about twice the float precision.
__device__ __forceinline__ void comp_term(float& s, float& c, float n, float v)
{
    const float p = __fmul_rn(n, v);
    const float e = __fmaf_rn(n, v, -p);
    const float t = __fadd_rn(s, p);
    const float err = fabsf(s) >= fabsf(p) ? __fadd_rn(__fadd_rn(s, -t), p)
                                           : __fadd_rn(__fadd_rn(p, -t), s);
    s = t;
    c = __fadd_rn(c, __fadd_rn(err, e));
}

// One CTA per SM: its tile into shared memory, then its groups, each warp
// taking the next one.  A lane's words come U at a time, the next U asked for
// before these are used; the first words of the next group and the head of
// the one after it are asked for before this group is summed (most groups are
// only a few U long, so a group's own start would wait for memory each time).
// Bound: the edge words' way from HBM (4.5 TB/s over the whole sweep).  U = 4
// and 6 were slower (111 and 95 us against 87 on the forest), 10 equal; a
// queue of groups shared by the CTAs of a tile, longest first or in order, 100-125.
// kComp: compensated sums, two floats per partial.
template <bool kComp>
__global__ void __launch_bounds__(kThreads, 1) k_gather(View v, const float* B,
                                                        float* __restrict__ partial,
                                                        const uint32_t* done)
{
    extern __shared__ __align__(16) float tile[];
    start_next();
    const uint32_t lane = threadIdx.x & 31;
    // The plan's own arrays first: no kernel that may still run writes them.
    const Share p = v.shares[blockIdx.x];
    const uint32_t at = p.tile * kTile, m = min(kTile, v.surfaces - at);
    __shared__ uint32_t queue;
    if (threadIdx.x == 0) queue = kThreads / 32;
    uint32_t g = p.begin + threadIdx.x / 32;
    const size_t out = size_t(p.tile) * v.surfaces;
    constexpr int U = 8;
    uint32_t meta = 0, meta1 = 0;          // heads of this group and the next
    uint2 info = make_uint2(0, 0), info1 = info;
    if (g < p.end) {
        meta = __ldcs(v.meta + size_t(g) * 32 + lane);
        info = __ldcs(v.groups + g);
    }
    auto take = [&] {
        uint32_t k = 0;
        if (lane == 0) k = p.begin + atomicAdd(&queue, 1u);
        return __shfl_sync(0xffffffffu, k, 0);
    };
    uint32_t x[U], z[U];
    uint32_t n = __reduce_max_sync(0xffffffffu, meta >> 16);  // words of the group's longest row
    const uint32_t* w = v.words + size_t(info.x) * 32 + lane;
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (uint32_t(u) < n) x[u] = __ldcs(w + u * 32);
    wait_for_previous();
    if (done && *done) return;
    for (uint32_t i = threadIdx.x; i < m / 4; i += kThreads) cp_async16(tile + 4 * i, B + at + 4 * i);
    if (threadIdx.x < (m & 3)) tile[(m & ~3u) + threadIdx.x] = B[at + (m & ~3u) + threadIdx.x];
    cp_commit();
    if (threadIdx.x == 0) tile[kPad] = 0.0f;
    __syncthreads();  // the queue's start
    uint32_t g1 = take();
    if (g1 < p.end) {
        meta1 = __ldcs(v.meta + size_t(g1) * 32 + lane);
        info1 = __ldcs(v.groups + g1);
    }
    cp_wait<0>();
    __syncthreads();
    while (g < p.end) {
        const uint32_t len = meta >> 16, row = info.y + (meta & 0xffffu);
        // the first words of the next group and the head of the one after it
        const uint32_t n1 = __reduce_max_sync(0xffffffffu, meta1 >> 16);
        const uint32_t* w1 = v.words + size_t(info1.x) * 32 + lane;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (uint32_t(u) < n1) z[u] = __ldcs(w1 + u * 32);
        g = g1;
        meta = meta1;
        info = info1;
        g1 = take();
        meta1 = 0;
        if (g1 < p.end) {
            meta1 = __ldcs(v.meta + size_t(g1) * 32 + lane);
            info1 = __ldcs(v.groups + g1);
        }
        float s = 0.0f, c = 0.0f;
        auto add = [&](uint32_t word) {
            const float count = __uint_as_float(word & 0xffff0000u);
            const float b = tile[word & 0xffffu];
            if (kComp) comp_term(s, c, count, b);
            else s += count * b;
        };
        uint32_t k = 0;
        for (; k + 2 * U <= n; k += U) {
            w += U * 32;
            uint32_t y[U];
#pragma unroll
            for (int u = 0; u < U; ++u) y[u] = __ldcs(w + u * 32);
#pragma unroll
            for (int u = 0; u < U; ++u) add(x[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) x[u] = y[u];
        }
        if (k + U < n) {
            w += U * 32;
            uint32_t y[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k + U + u < n) y[u] = __ldcs(w + u * 32);
#pragma unroll
            for (int u = 0; u < U; ++u) add(x[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k + U + u < n) add(y[u]);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k + u < n) add(x[u]);
        }
        if (len) {
            if (kComp) reinterpret_cast<float2*>(partial)[out + row] = make_float2(s, c);
            else partial[out + row] = s;
        }
        n = n1;
        w = w1;
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = z[u];
    }
}

__device__ __forceinline__ float2 sum_pair(const float* partial, uint32_t tiles, uint32_t S,
                                           uint32_t f)
{
    float2 a = make_float2(0.0f, 0.0f);
    for (uint32_t t = 0; t < tiles; ++t) {
        const float2 q = *reinterpret_cast<const float2*>(partial + size_t(t) * S + 2 * f);
        a.x += q.x;
        a.y += q.y;
    }
    return a;
}

// A thread per facet: the reference's update (as k_jacobi_rows in solve.cu).
__global__ void __launch_bounds__(256) k_finish_jacobi(
    uint32_t facets, uint32_t tiles, const float* partial, const uint2* __restrict__ denom,
    const uint2* __restrict__ skyc, const float4* optics, float sky, float relax,
    const float2* in, float2* out, uint32_t* max_delta_bits)
{
    start_next();
    wait_for_previous();
    __shared__ float block_delta[8];
    const uint32_t f = blockIdx.x * 256 + threadIdx.x;
    float delta = 0.0f;
    if (f < facets) {
        const uint2 d = denom[f], sk = skyc[f];
        const float4 o0 = optics[2 * size_t(f)], o1 = optics[2 * size_t(f) + 1];  // rho, tau, e, D
        const float2 old = in[f];
        const float2 a = sum_pair(partial, tiles, 2 * facets, f);
        const float h0 = (d.x ? (float(sk.x) * sky + a.x) / float(d.x) : sky) + o0.w;
        const float h1 = (d.y ? (float(sk.y) * sky + a.y) / float(d.y) : sky) + o1.w;
        const float t0 = o0.z + o0.x * h0 + o0.y * h1;
        const float t1 = o1.z + o1.x * h1 + o1.y * h0;
        // GLSL mix(x, y, a) = x * (1 - a) + y * a
        const float n0 = old.x * (1.0f - relax) + t0 * relax;
        const float n1 = old.y * (1.0f - relax) + t1 * relax;
        out[f] = make_float2(n0, n1);
        delta = fmaxf(fabsf(n0 - old.x), fabsf(n1 - old.y));
    }
    for (int k = 16; k > 0; k >>= 1) delta = fmaxf(delta, __shfl_xor_sync(0xffffffffu, delta, k));
    if ((threadIdx.x & 31) == 0) block_delta[threadIdx.x >> 5] = delta;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) delta = fmaxf(delta, block_delta[w]);
        atomicMax(max_delta_bits, __float_as_uint(delta));
    }
}

// A thread per facet: the batched solver's update and statistics (as
// k_sweep<1> in batched.cu); in == nullptr stands for zeros.
__global__ void __launch_bounds__(256) k_finish_panel(
    uint32_t facets, uint32_t tiles, const float* partial, const uint2* __restrict__ denom,
    const uint2* __restrict__ skyc, const float2* rho, const float2* tau, const float2* emis,
    const float2* direct, const float* skyL, const float* colmax, const float2* in, float2* out,
    uint32_t* stats, const uint32_t* done)
{
    start_next();
    wait_for_previous();
    if (*done) return;
    __shared__ float red[3][8];
    const uint32_t f = blockIdx.x * 256 + threadIdx.x;
    float m[3] = {0.0f, 0.0f, 0.0f};  // max|dB|, max|B|, worst per-side change
    if (f < facets) {
        const float L = skyL[0], floor_abs = kSideFloor * colmax[0];
        const uint2 d = denom[f], sk = skyc[f];
        const float2 r = rho[f], ta = tau[f], e = emis[f], dir = direct[f];
        const float2 o = in ? in[f] : make_float2(0.0f, 0.0f);
        const float2 a = sum_pair(partial, in ? tiles : 0u, 2 * facets, f);
        const float h0 = (d.x ? (float(sk.x) * L + a.x) / float(d.x) : L) + dir.x;
        const float h1 = (d.y ? (float(sk.y) * L + a.y) / float(d.y) : L) + dir.y;
        const float b0 = e.x + r.x * h0 + ta.x * h1;
        const float b1 = e.y + r.y * h1 + ta.y * h0;
        out[f] = make_float2(b0, b1);
        m[0] = fmaxf(fabsf(b0 - o.x), fabsf(b1 - o.y));
        m[1] = fmaxf(fabsf(b0), fabsf(b1));
        m[2] = fmaxf(rel_change(b0 - o.x, b0, floor_abs), rel_change(b1 - o.y, b1, floor_abs));
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        for (int k = 16; k > 0; k >>= 1) m[q] = fmaxf(m[q], __shfl_xor_sync(0xffffffffu, m[q], k));
        if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = m[q];
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        float x = red[threadIdx.x][0];
        for (int w = 1; w < 8; ++w) x = fmaxf(x, red[threadIdx.x][w]);
        atomicMax(stats + threadIdx.x * kMaxP, __float_as_uint(x));
    }
}

// A thread per side: max(0, incident diffuse radiation) from compensated
// partials (the FacetEB node).
__global__ void __launch_bounds__(256) k_finish_incident(
    uint32_t S, uint32_t tiles, const float2* partial, const uint32_t* __restrict__ denom,
    const uint32_t* __restrict__ skyc, const float* sky, float* out)
{
    start_next();
    wait_for_previous();
    const uint32_t s = blockIdx.x * 256 + threadIdx.x;
    if (s >= S) return;
    const float L = sky[0];
    const uint32_t d = denom[s];
    float h = L;
    if (d) {
        Csum sum{0.0f, 0.0f};
        for (uint32_t t = 0; t < tiles; ++t) {
            const float2 q = partial[size_t(t) * S + s];
            csum_add(sum, q.x, q.y);
        }
        h = diffuse_mean(sum, skyc[s], L, d);
    }
    out[s] = (0.0f < h) ? h : 0.0f;
}

float2* compensated(const DeviceGraph& g)
{
    return reinterpret_cast<float2*>(g.column.partial.as<float>() +
                                     size_t(g.column.tiles) * g.surfaces);
}

// The gathers and what finishes them follow one another without the 2 us
// between two launches: each starts while the one before it ends and waits
// inside, the gather with its plan's first words in registers (64 sweeps of the
// 200,000-facet forest 6.91 -> 6.63 ms).  The arrays that a kernel before writes
// are not __restrict__, so that no load of them moves above the wait.
template <bool kComp>
void gather(const DeviceGraph& g, const float* B, const uint32_t* done, cudaStream_t s)
{
    const ColumnPlan& c = g.column;
    const View v{c.shares.as<Share>(), c.groups.as<uint2>(), c.meta.as<uint32_t>(),
                 c.words.as<uint32_t>(), c.tiles, g.surfaces};
    const int smem = int((kTile + 1u) * 4u);
    FCU_CHECK(cudaFuncSetAttribute(k_gather<kComp>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   smem));
    float* partial = kComp ? reinterpret_cast<float*>(compensated(g)) : c.partial.as<float>();
    launch_early(k_gather<kComp>, c.ctas, kThreads, smem, s, v, B, partial, done);
}

bool make_plan(DeviceGraph& g, Workspace& ws, cudaStream_t s)
{
    ColumnPlan& c = g.column;
    const uint32_t S = g.surfaces;
    if (S < 2 || g.nnz < kMinEdges || g.max_count > kMaxCount) return false;
    const uint32_t tiles = (S + kTile - 1) / kTile;
    if (tiles > kMaxTiles || g.nnz < kMinTileEdges * tiles * S) return false;
    const uint32_t windows = (S + kWindow - 1) / kWindow;
    const uint32_t cells = tiles * windows;
    const uint32_t* rows = g.row_offsets.as<uint32_t>();
    const uint32_t* packed = g.packed_valid ? g.packed.as<uint32_t>() : nullptr;
    const facetcu_csr_edge* edges = g.edges.as<facetcu_csr_edge>();

    ScratchBuffer seg_buf(ws), slot_buf(ws), ng_buf(ws), first_buf(ws), group_buf(ws);
    uint16_t* seg = static_cast<uint16_t*>(seg_buf.reserve(size_t(tiles) * S * 2));
    uint16_t* slot = static_cast<uint16_t*>(slot_buf.reserve(size_t(tiles) * S * 2));
    uint32_t* ng = static_cast<uint32_t*>(ng_buf.reserve(size_t(cells) * 4));
    uint32_t* first = static_cast<uint32_t*>(first_buf.reserve((size_t(cells) + 1) * 4));
    unsigned long long* total = static_cast<unsigned long long*>(ws.e.reserve(64));
    uint32_t* longest = reinterpret_cast<uint32_t*>(total + 1);
    FCU_CHECK(cudaMemsetAsync(total, 0, 16, s));
    // slots of pairs without edges are read (and not used)
    FCU_CHECK(cudaMemsetAsync(slot, 0, size_t(tiles) * S * 2, s));
    k_count<<<blocks(S, 8), 256, 0, s>>>(rows, packed, edges, g.nb_bits, S, tiles, seg, longest);
    FCU_LAUNCH("k_count");
    k_groups<<<cells, 256, 0, s>>>(S, windows, seg, ng);
    FCU_LAUNCH("k_groups");
    exclusive_scan_u32(ng, first, cells, total, ws, s);
    std::vector<uint32_t> host_first(cells);
    unsigned long long host[2] = {0, 0};
    FCU_CHECK(cudaMemcpyAsync(host, total, 16, cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaMemcpyAsync(host_first.data(), first, size_t(cells) * 4, cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaStreamSynchronize(s));
    const size_t slots = size_t(host[0]);
    if (uint32_t(host[1]) || slots == 0) return false;
    std::vector<uint32_t> tile_group(tiles + 1, uint32_t(slots)), tile_word(tiles + 1);
    for (uint32_t t = 0; t < tiles; ++t) tile_group[t] = host_first[size_t(t) * windows];
    // per group: words of its longest row, first word (a row without edges may
    // read woff[slots])
    uint32_t* glen = static_cast<uint32_t*>(group_buf.reserve((slots * 2 + tiles + 2) * 4));
    uint32_t* woff = glen + slots;
    uint32_t* d_tile_group = woff + slots + 1;
    uint32_t* meta = static_cast<uint32_t*>(c.meta.reserve(slots * 128));
    FCU_CHECK(cudaMemcpyAsync(d_tile_group, tile_group.data(), (tiles + 1) * 4,
                              cudaMemcpyHostToDevice, s));
    k_order<<<cells, 256, 0, s>>>(S, windows, seg, first, slot, meta, glen);
    FCU_LAUNCH("k_order");
    exclusive_scan_u32(glen, woff, slots, total, ws, s);
    k_group_info<<<cells, 128, 0, s>>>(windows, first, ng, woff,
                                       static_cast<uint2*>(c.groups.reserve(slots * 8)));
    FCU_LAUNCH("k_group_info");
    FCU_CHECK(cudaMemcpyAsync(host, total, 8, cudaMemcpyDeviceToHost, s));
    for (uint32_t t = 0; t < tiles; ++t)
        if (tile_group[t] < slots)
            FCU_CHECK(cudaMemcpyAsync(&tile_word[t], woff + tile_group[t], 4,
                                      cudaMemcpyDeviceToHost, s));
    FCU_CHECK(cudaStreamSynchronize(s));
    // padding: a group is as long as its longest row (a few per cent where
    // the rows of a window vary as usual); give up where it doubles the words
    const unsigned long long words32 = host[0];
    if (words32 * 32 > 2 * g.nnz + 32 * slots || words32 > 0xffffffffull) return false;
    for (uint32_t t = 0; t <= tiles; ++t)
        if (tile_group[t] >= slots) tile_word[t] = uint32_t(words32);

    // CTAs per tile: one each, then always to the tile with the most work per CTA
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    std::vector<uint64_t> work(tiles);
    std::vector<uint32_t> share(tiles, 0);
    uint32_t ctas = 0;
    for (uint32_t t = 0; t < tiles; ++t) {
        work[t] = uint64_t(tile_word[t + 1] - tile_word[t]) +
                  uint64_t(kGroupCost) * (tile_group[t + 1] - tile_group[t]);
        if (work[t]) ctas += share[t] = 1;
    }
    while (ctas < uint32_t(std::max(sms, 1))) {
        uint32_t best = 0;
        double most = -1.0;
        for (uint32_t t = 0; t < tiles; ++t)
            if (share[t] && double(work[t]) / share[t] > most) {
                most = double(work[t]) / share[t];
                best = t;
            }
        ++share[best];
        ++ctas;
    }
    std::vector<Share> shares;
    for (uint32_t t = 0; t < tiles; ++t)
        for (uint32_t k = 0; k < share[t]; ++k) shares.push_back({t, k, share[t]});
    Share* d_shares = static_cast<Share*>(c.shares.reserve(2 * ctas * sizeof(Share))) + ctas;
    FCU_CHECK(cudaMemcpyAsync(d_shares, shares.data(), ctas * sizeof(Share), cudaMemcpyHostToDevice, s));
    k_split<<<blocks(ctas, 128), 128, 0, s>>>(woff, uint32_t(slots), uint32_t(words32), d_shares,
                                              d_tile_group, ctas, c.shares.as<Share>());
    FCU_LAUNCH("k_split");
    uint32_t* words = static_cast<uint32_t*>(c.words.reserve(size_t(words32) * 128));
    k_fill<<<blocks(size_t(words32) * 8, 256), 256, 0, s>>>(reinterpret_cast<uint4*>(words),
                                                            size_t(words32) * 8);
    FCU_LAUNCH("k_fill");
    k_scatter<<<blocks(S, 8), 256, 0, s>>>(rows, packed, edges, g.nb_bits, S, tiles, windows, first,
                                           slot, woff, words);
    FCU_LAUNCH("k_scatter");
    // [tiles][S] sums, then [tiles][S] compensated ones; pairs without edges
    // keep their zeros
    const size_t partial = size_t(tiles) * S * 12;
    FCU_CHECK(cudaMemsetAsync(c.partial.reserve(partial), 0, partial, s));
    FCU_CHECK(cudaStreamSynchronize(s));  // the tables go out of scope
    c.ctas = ctas;
    c.tiles = tiles;
    return true;
}

}  // namespace

void ColumnPlan::release()
{
    for (DeviceBuffer* b : {&shares, &groups, &meta, &words, &partial}) b->release();
    state = kUnknown;
}

// Sweeps from which a first solve, the making of the plan included, is not slower
// than over the CSR.  Making it takes some 0.35 ms and 14 us a million edges; a
// sweep saves 9.5 us of 40 at 15.9 M edges and 77 of 160 at 83.8 M.  A first call
// in ms, with the plan and without:
//     sweeps          8           16          24          32          48          64
//     15.9 M edges    1.15  0.70  1.37  1.00  1.61  1.32  1.85  1.62  2.28  2.25  2.75  2.87
//     22.0 M          1.46  0.94  1.69  1.32  1.95  1.75  2.20  2.14  2.72  2.95  3.24  3.79
//     37.4 M          1.96  1.35  2.33  2.01  2.68  2.62  3.00  3.28  3.72  4.53  4.38  5.81
//     83.8 M          3.49  2.62  4.14  3.90  4.83  5.17  5.47  6.46  6.80  9.01  8.15  11.6
// so the two meet at about 50, 36, 26 and 20 sweeps; the line says 46, 37, 27 and 19,
// and 64 from the fewest edges that get a plan.
bool column_plan_pays(const DeviceGraph& g, uint32_t sweeps)
{
    return sweeps >= 12u && g.nnz * (sweeps - 12u) >= 540000000ull;
}

bool column_plan(DeviceGraph& g, Workspace& ws, cudaStream_t s)
{
    ColumnPlan& c = g.column;
    if (c.state == ColumnPlan::kUnknown) {
        bool made = false;
        try {
            made = make_plan(g, ws, s);
        } catch (const Error& e) {
            if (e.code != FACETCU_OUT_OF_MEMORY) throw;  // the CSR sweeps need no extra memory
        }
        if (!made) c.release();
        c.state = made ? ColumnPlan::kMade : ColumnPlan::kNone;
    }
    return c.state == ColumnPlan::kMade;
}

void column_jacobi(const DeviceGraph& g, const facetcu_surface_optics* optics, float sky,
                   float relax, const float* in, float* out, uint32_t* max_delta_bits,
                   cudaStream_t s)
{
    const uint32_t facets = g.surfaces / 2;
    gather<false>(g, in, nullptr, s);
    launch_early(k_finish_jacobi, blocks(facets, 256), 256, 0, s, facets, g.column.tiles,
                 g.column.partial.as<float>(), g.denominators.as<uint2>(), g.sky.as<uint2>(),
                 reinterpret_cast<const float4*>(optics), sky, relax,
                 reinterpret_cast<const float2*>(in), reinterpret_cast<float2*>(out),
                 max_delta_bits);
}

void column_sweep(const DeviceGraph& g, const float* rho, const float* tau, const float* emis,
                  const float* direct, const float* skyL, const float* colmax, const float* in,
                  float* out, uint32_t* stats, const uint32_t* done, cudaStream_t s)
{
    const uint32_t facets = g.surfaces / 2;
    if (in) gather<false>(g, in, done, s);
    auto pair = [](const float* p) { return reinterpret_cast<const float2*>(p); };
    launch_early(k_finish_panel, blocks(facets, 256), 256, 0, s, facets, g.column.tiles,
                 g.column.partial.as<float>(), g.denominators.as<uint2>(), g.sky.as<uint2>(),
                 pair(rho), pair(tau), pair(emis), pair(direct), skyL, colmax, pair(in),
                 reinterpret_cast<float2*>(out), stats, done);
}

void column_incident(const DeviceGraph& g, const float* B, const float* sky, float* out,
                     cudaStream_t s)
{
    gather<true>(g, B, nullptr, s);
    launch_early(k_finish_incident, blocks(g.surfaces, 256), 256, 0, s, g.surfaces, g.column.tiles,
                 compensated(g), g.denominators.as<uint32_t>(), g.sky.as<uint32_t>(), sky, out);
}

}  // namespace facetcu
