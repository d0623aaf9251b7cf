// image.cu — sensor images of per-side values (the reference's
// writeRadiosityTiffForAngle, server.mjs:1127-1600, a JavaScript routine of
// its Node backend that runs on the host, pixel loop by pixel loop).
//
// Here the raster runs on the device:
//   k_raster    per facet: its three vertices projected to the sensor
//               (viewVertex :1295-1307), the side it shows (:1309-1317) and
//               its pixel box; the barycentric test at pixel centres
//               (:1335-1347); per pixel the nearest depth, and among equal
//               depths the smallest facet index, i.e. the facet the
//               reference's sequential loop keeps (it replaces a pixel only
//               for a strictly nearer depth)
//   k_raster_large  the same for the facets with large boxes
//   k_observed  facet -> observed side index image
//   k_nadir     a parallel sensor's output grid mapped back into the
//               observed image (:1363-1387)
//   k_fill      per band and pixel: the side's value, else for a
//               perspective sensor the analytic sky (skyOutputValue
//               :1229-1255, no atmosphere table), else NaN
// Every coordinate is a double, computed in the reference's operation order
// (this file is compiled with -fmad=false), so the side index image is the
// reference's arithmetic exactly.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "internal.h"

namespace facetcu {
namespace image {
namespace {

__device__ __forceinline__ double ddot(const double* a, const double* b)
{
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

struct Proj {
    double x, y, depth;
    int valid;
};

__device__ Proj project(const Camera& c, const double* p)
{
    Proj r;
    if (!c.perspective) {
        r.x = (ddot(p, c.right) - c.min_x) / c.range_x * double(c.width);
        r.y = (c.max_y - ddot(p, c.up)) / c.range_y * double(c.height);
        r.depth = ddot(p, c.out);
        r.valid = 1;
        return r;
    }
    const double rel[3] = {p[0] - c.cam_pos[0], p[1] - c.cam_pos[1], p[2] - c.cam_pos[2]};
    const double depth = ddot(rel, c.forward);
    const double half_w = c.tan_half * double(c.width) / double(c.height);
    r.x = (0.5 + ddot(rel, c.right) / (2.0 * depth * half_w)) * double(c.width);
    r.y = (0.5 - ddot(rel, c.up) / (2.0 * depth * c.tan_half)) * double(c.height);
    r.depth = -depth;
    r.valid = depth > 1e-6 ? 1 : 0;
    return r;
}

__device__ __forceinline__ double edge_fn(const Proj& a, const Proj& b, double x, double y)
{
    return (x - a.x) * (b.y - a.y) - (y - a.y) * (b.x - a.x);
}

__device__ __forceinline__ unsigned long long depth_key(double d)
{
    const long long b = __double_as_longlong(d);
    return b >= 0 ? (static_cast<unsigned long long>(b) | 0x8000000000000000ull)
                  : ~static_cast<unsigned long long>(b);
}

// The nearest fragment of a pixel, {depth key, 2^32 - 1 - facet} as one
// 16-byte value that only grows (both 0: nothing seen).
__device__ __forceinline__ ulonglong2 cas16(ulonglong2* p, ulonglong2 expected, ulonglong2 value)
{
    ulonglong2 old;
    asm volatile(
        "{ .reg .b128 e, v, o;\n"
        "  mov.b128 e, {%2, %3};\n"
        "  mov.b128 v, {%4, %5};\n"
        "  atom.global.cas.b128 o, [%6], e, v;\n"
        "  mov.b128 {%0, %1}, o; }"
        : "=l"(old.x), "=l"(old.y)
        : "l"(expected.x), "l"(expected.y), "l"(value.x), "l"(value.y), "l"(p)
        : "memory");
    return old;
}

__device__ __forceinline__ void keep_nearest(ulonglong2* p, double depth, uint32_t f)
{
    const ulonglong2 mine = make_ulonglong2(depth_key(depth), 0xffffffffull - f);
    // A plain read first: keys only grow, so a larger one settles it.  Its two
    // halves may come from different writes, so nothing else is decided on it.
    ulonglong2 cur = __ldcg(p);
    if (mine.x < cur.x) return;
    if (mine.x == cur.x) cur = cas16(p, cur, cur);  // both halves as they are
    while (mine.x > cur.x || (mine.x == cur.x && mine.y > cur.y)) {
        const ulonglong2 old = cas16(p, cur, mine);
        if (old.x == cur.x && old.y == cur.y) return;
        cur = old;
    }
}

// A projected facet and its pixel box.  The double test decides; before it a
// float test of the three edges, relative to the box, rejects the pixels that
// are outside by more than its rounding can account for.  FP64 is what bounds
// this (GB300 has two lanes per SM and clock): the reference's test costs two
// divisions and about twenty other operations.
struct Tri {
    Proj a, b, c;
    double area;
    int x0, y0;
    uint32_t w, h;            // pixel box; 0: nothing to cover
    float ax, ay, bx, by, cx, cy, sign, tol;
};

__device__ __forceinline__ void make_box(const Camera& c, Tri& t)
{
    t.w = t.h = 0;
    if (!t.a.valid || !t.b.valid || !t.c.valid) return;
    t.area = edge_fn(t.a, t.b, t.c.x, t.c.y);
    if (fabs(t.area) < 1e-10) return;
    const double W = double(c.width), H = double(c.height);
    const double x0 = fmax(0.0, floor(fmin(fmin(t.a.x, t.b.x), t.c.x)));
    const double x1 = fmin(W - 1.0, ceil(fmax(fmax(t.a.x, t.b.x), t.c.x)) - 1.0);
    const double y0 = fmax(0.0, floor(fmin(fmin(t.a.y, t.b.y), t.c.y)));
    const double y1 = fmin(H - 1.0, ceil(fmax(fmax(t.a.y, t.b.y), t.c.y)) - 1.0);
    if (!(x1 >= x0) || !(y1 >= y0)) return;
    t.x0 = int(x0);
    t.y0 = int(y0);
    t.w = uint32_t(x1 - x0) + 1u;
    t.h = uint32_t(y1 - y0) + 1u;
    t.ax = float(t.a.x - x0), t.ay = float(t.a.y - y0);
    t.bx = float(t.b.x - x0), t.by = float(t.b.y - y0);
    t.cx = float(t.c.x - x0), t.cy = float(t.c.y - y0);
    t.sign = t.area > 0.0 ? 1.0f : -1.0f;
    // M bounds every coordinate; an edge function's float error is below
    // 40 2^-24 M^2, and the tolerance of the double test, 1e-7 |area|, below
    // 4e-7 M^2: 2^-17 M^2 covers both.  (Not finite: nothing is rejected.)
    const float m0 = fmaxf(fmaxf(fabsf(t.ax), fabsf(t.ay)), fmaxf(fabsf(t.bx), fabsf(t.by)));
    const float m1 = fmaxf(fmaxf(fabsf(t.cx), fabsf(t.cy)), fmaxf(float(t.w), float(t.h)));
    const float M = fmaxf(m0, m1);
    t.tol = 7.62939453125e-6f * M * M;
}

__device__ __forceinline__ void test_pixel(const Camera& c, const Tri& t, uint32_t i, uint32_t j,
                                           uint32_t f, ulonglong2* zbuf)
{
    const float px = float(i) + 0.5f, py = float(j) + 0.5f;
    const float ea = (px - t.bx) * (t.cy - t.by) - (py - t.by) * (t.cx - t.bx);
    const float eb = (px - t.cx) * (t.ay - t.cy) - (py - t.cy) * (t.ax - t.cx);
    const float ec = (px - t.ax) * (t.by - t.ay) - (py - t.ay) * (t.bx - t.ax);
    if (ea * t.sign < -t.tol || eb * t.sign < -t.tol || ec * t.sign < -t.tol) return;
    const double sx = double(t.x0) + double(i) + 0.5, sy = double(t.y0) + double(j) + 0.5;
    const double wa = edge_fn(t.b, t.c, sx, sy) / t.area;
    const double wb = edge_fn(t.c, t.a, sx, sy) / t.area;
    const double wc = 1.0 - wa - wb;
    if (wa < -1e-7 || wb < -1e-7 || wc < -1e-7) return;
    const double depth = wa * t.a.depth + wb * t.b.depth + wc * t.c.depth;
    keep_nearest(zbuf + size_t(t.y0 + int(j)) * c.width + size_t(t.x0 + int(i)), depth, f);
}

__device__ __forceinline__ void load_facet(const facetcu_vertex* __restrict__ V, uint32_t f,
                                           double (&p)[3][3])
{
    for (int k = 0; k < 3; ++k)
        for (int a = 0; a < 3; ++a) p[k][a] = double(V[3 * size_t(f) + k].position[a]);
}
__device__ __forceinline__ void project_facet(const Camera& c, const double (&p)[3][3], Tri& t)
{
    t.a = project(c, p[0]);
    t.b = project(c, p[1]);
    t.c = project(c, p[2]);
    make_box(c, t);
}

// A lane per facet projects it and, for a box of at most kSmallBox pixels,
// tests them; the warp then takes its larger facets one by one, a lane per
// pixel.  (A warp per facet did the projection's and the box's doubles in all
// lanes, and two passes over the pixels, depth and index, did the test twice:
// 2.29 ms for 200,000 facets on 1,024 x 1,024 pixels, 0.49 here.)  What a warp
// does in turn is bounded twice: it takes `per_warp` facets, fewer than 32 where
// there would be too few warps (render), and boxes above kLargeBox are listed for
// k_raster_large.  A side image of 1,024 x 1,024, copy included, in ms with a warp
// per facet and box / 32 facets a warp / so:
//     2 ground triangles        107    80.5   0.31
//     64 facets of some metres  10.1   33.5   0.33
//     288 soil triangles        1.77   14.3   0.39
//     4,096 facets              0.76   2.0    0.43
//     20,000 panels of 0.6 m    10.4   8.3    4.7
//     200,000 facets            2.69   0.98   0.81
// (Six blocks an SM, a few spilled words: without them the list cost the last row
// 1.5 %.)
constexpr uint32_t kSmallBox = 16, kLargeBox = 1024;
constexpr int kRasterThreads = 128;
__global__ void __launch_bounds__(kRasterThreads, 6) k_raster(
    uint32_t F, uint32_t per_warp, const facetcu_vertex* __restrict__ V, Camera c,
    ulonglong2* __restrict__ zbuf, int32_t* __restrict__ side, uint32_t* __restrict__ large_list,
    uint32_t* large_count)
{
    __shared__ Tri large[kRasterThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t f = (blockIdx.x * (kRasterThreads / 32) + warp) * per_warp + lane;
    Tri t;
    t.w = t.h = 0;
    if (lane < per_warp && f < F) {
        double p[3][3];
        load_facet(V, f, p);
        const double e1[3] = {p[1][0] - p[0][0], p[1][1] - p[0][1], p[1][2] - p[0][2]};
        const double e2[3] = {p[2][0] - p[0][0], p[2][1] - p[0][1], p[2][2] - p[0][2]};
        const double n[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2],
                             e1[0] * e2[1] - e1[1] * e2[0]};
        double d[3];
        if (c.perspective) {
            for (int a = 0; a < 3; ++a) d[a] = c.cam_pos[a] - (p[0][a] + p[1][a] + p[2][a]) / 3.0;
        } else {
            for (int a = 0; a < 3; ++a) d[a] = c.out[a];
        }
        side[f] = int32_t(2 * f + (ddot(n, d) >= 0.0 ? 0 : 1));
        project_facet(c, p, t);
    }
    const unsigned long long pixels = (unsigned long long)t.w * t.h;
    if (pixels <= kSmallBox) {
        for (uint32_t j = 0; j < t.h; ++j)
            for (uint32_t i = 0; i < t.w; ++i) test_pixel(c, t, i, j, f, zbuf);
    }
    if (pixels > kLargeBox) {
        large_list[atomicAdd(large_count, 1u)] = f;
        t.w = t.h = 0;
    }
    uint32_t todo = __ballot_sync(0xffffffffu, t.w * t.h > kSmallBox);
    while (todo) {
        const int from = __ffs(int(todo)) - 1;
        todo &= todo - 1u;
        if (int(lane) == from) large[warp] = t;
        __syncwarp();
        const Tri& q = large[warp];
        const uint32_t facet = __shfl_sync(0xffffffffu, f, from);
        const uint32_t w = q.w, h = q.h, dx = 32u % w, dy = 32u / w;
        uint32_t i = lane % w, j = lane / w;
        while (j < h) {
            test_pixel(c, q, i, j, facet, zbuf);
            i += dx;
            j += dy;
            if (i >= w) {
                i -= w;
                ++j;
            }
        }
        __syncwarp();
    }
}

// The listed facets: with few of them the blocks share a facet, taking parts of
// kPartPixels pixels of its box in turn; with more than blocks each takes whole
// ones (the projection is done once a block and facet).  Bound by FP64, as k_raster.
constexpr uint32_t kPartPixels = 2048;
__global__ void __launch_bounds__(256) k_raster_large(const facetcu_vertex* __restrict__ V, Camera c,
                                                      ulonglong2* __restrict__ zbuf,
                                                      const uint32_t* large_list,
                                                      const uint32_t* large_count)
{
    __shared__ Tri t;
    const uint32_t count = *large_count;
    if (!count) return;
    const uint32_t share = max(1u, gridDim.x / count);  // blocks of a facet
    const uint32_t part = blockIdx.x % share;
    for (uint32_t k = blockIdx.x / share; k < count; k += (gridDim.x + share - 1u) / share) {
        const uint32_t f = large_list[k];
        if (threadIdx.x == 0) {
            double p[3][3];
            Tri mine;
            load_facet(V, f, p);
            project_facet(c, p, mine);
            t = mine;
        }
        __syncthreads();
        // (at most 2^28 pixels an image)
        const uint32_t pixels = t.w * t.h, w = t.w, dx = 256u % w, dy = 256u / w;
        for (uint32_t first = part * kPartPixels; first < pixels; first += share * kPartPixels) {
            const uint32_t end = min(pixels, first + kPartPixels);
            uint32_t i = (first + threadIdx.x) % w, j = (first + threadIdx.x) / w;
            for (uint32_t q = first + threadIdx.x; q < end; q += 256) {
                test_pixel(c, t, i, j, f, zbuf);
                i += dx;
                j += dy;
                if (i >= w) {
                    i -= w;
                    ++j;
                }
            }
        }
        __syncthreads();  // t is free again
    }
}

__global__ void k_observed(size_t n, const ulonglong2* __restrict__ zbuf,
                           const int32_t* __restrict__ side, int32_t* __restrict__ img,
                           uint32_t* __restrict__ count)
{
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t low = uint32_t(zbuf[i].y);
    const bool seen = low != 0u;
    img[i] = seen ? side[0xffffffffu - low] : -1;
    const unsigned active = __activemask();
    const unsigned m = __ballot_sync(active, seen);
    if ((threadIdx.x & 31u) == unsigned(__ffs(active) - 1)) atomicAdd(count, unsigned(__popc(m)));
}

// A block takes 32 x 8 output pixels: what depends on the row or the column
// alone (a division and the row's or column's part of both dot products, in
// the reference's order of additions) is computed once for each.
__global__ void __launch_bounds__(256) k_nadir(Camera c, const int32_t* __restrict__ observed,
                                               int32_t* __restrict__ out,
                                               uint32_t* __restrict__ count)
{
    __shared__ double row_right[8], row_up[8], col_right[32], col_up[32];
    __shared__ bool row_in[8], col_in[32];
    const uint32_t across = (c.width + 31) / 32;
    const uint32_t x0 = blockIdx.x % across * 32, y0 = blockIdx.x / across * 8;
    const uint32_t x = x0 + (threadIdx.x & 31), y = y0 + (threadIdx.x >> 5);
    if (threadIdx.x < 8) {
        const double rh = double(c.height > 1 ? c.height - 1 : 1);
        const double wx = c.orth_max_x - double(y0 + threadIdx.x) / rh * c.orth_north;
        row_in[threadIdx.x] = !(wx < -c.scene_w / 2.0 || wx > c.scene_w / 2.0);
        row_right[threadIdx.x] = wx * c.right[0] + 0.0 * c.right[1];
        row_up[threadIdx.x] = wx * c.up[0] + 0.0 * c.up[1];
    } else if (threadIdx.x >= 32 && threadIdx.x < 64) {
        const uint32_t k = threadIdx.x - 32;
        const double rw = double(c.width > 1 ? c.width - 1 : 1);
        const double wz = c.orth_min_z + double(x0 + k) / rw * c.orth_east;
        col_in[k] = !(wz < -c.scene_d / 2.0 || wz > c.scene_d / 2.0);
        col_right[k] = wz * c.right[2];
        col_up[k] = wz * c.up[2];
    }
    __syncthreads();
    int32_t s = -1;
    const uint32_t i = threadIdx.x & 31, j = threadIdx.x >> 5;
    if (x < c.width && y < c.height) {
        if (row_in[j] && col_in[i]) {  // (a parallel sensor: project())
            const double px = (row_right[j] + col_right[i] - c.min_x) / c.range_x * double(c.width);
            const double py = (c.max_y - (row_up[j] + col_up[i])) / c.range_y * double(c.height);
            const double tx = trunc(px), ty = trunc(py);
            if (tx >= 0.0 && tx < double(c.width) && ty >= 0.0 && ty < double(c.height))
                s = observed[size_t(ty) * c.width + size_t(tx)];
        }
        out[size_t(y) * c.width + x] = s;
    }
    const unsigned m = __ballot_sync(0xffffffffu, s >= 0);
    if (i == 0 && m) atomicAdd(count, unsigned(__popc(m)));
}

__device__ double planck_js(double wl_nm, double temperature)
{
    const double um = wl_nm > 50.0 ? wl_nm / 1000.0 : wl_nm;
    return 1.19104e8 / (pow(um, 5.0) * expm1(14387.7 / (temperature * um)));
}

__device__ double inverse_planck_js(double wl_nm, double radiance)
{
    const double um = wl_nm > 50.0 ? wl_nm / 1000.0 : wl_nm;
    return 14387.7 / (um * log(1.19104e8 / (radiance * pow(um, 5.0)) + 1.0));
}

constexpr double kPiD = 3.141592653589793;

__device__ double sky_value(double wl_nm, double zenith_deg, bool as_temperature, double sky_t)
{
    const double wl = (wl_nm > 0.0 && wl_nm <= 50.0) ? wl_nm * 1000.0 : wl_nm;
    const double zr = fmax(0.0, fmin(89.5, zenith_deg)) * kPiD / 180.0;
    const double visibility = 23.0;
    if (wl <= 2500.0) {
        const double weight = fmax(0.06, fmin(2.0, pow(550.0 / fmax(350.0, fmin(2500.0, wl)), 1.8)));
        const double aerosol = fmax(0.4, fmin(2.3, 23.0 / visibility));
        const double cz = fmax(0.12, cos(zr));
        const double air_mass = 1.0 / cz;
        const double trans = exp(-(0.10 * weight + 0.025 * aerosol) * air_mass);
        const double boost = 1.0 + 0.55 * (1.0 - cz);
        return fmax(0.002, fmin(0.85, (1.0 - trans) * 0.55 * weight * boost + 0.008 * aerosol * boost));
    }
    const double cz = fmax(0.05, cos(zr));
    const double emis = 0.72;
    const double frac = fmax(emis, fmin(1.0, 1.0 - (1.0 - emis) * cz));
    const double radiance = planck_js(wl, sky_t) * frac;
    return as_temperature ? inverse_planck_js(wl, radiance) : radiance;
}

__global__ void k_fill(Camera c, uint32_t nb, size_t S, const int32_t* __restrict__ sides,
                       const float* __restrict__ values, const float* __restrict__ wavelengths,
                       int as_temperature, double sky_t, float* __restrict__ image)
{
    const size_t n = size_t(c.width) * c.height;
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n * nb) return;
    const uint32_t b = uint32_t(i / n);
    const size_t px = i % n;
    const int32_t s = sides[px];
    float v = __int_as_float(0x7fc00000);  // NaN
    if (s >= 0) {
        v = values[size_t(b) * S + size_t(s)];
    } else if (c.perspective) {
        const uint32_t x = uint32_t(px % c.width), y = uint32_t(px / c.width);
        const double vs = c.tan_half, hs = c.tan_half * double(c.width) / double(c.height);
        const double sy = (1.0 - 2.0 * (double(y) + 0.5) / double(c.height)) * vs;
        const double sx = (2.0 * (double(x) + 0.5) / double(c.width) - 1.0) * hs;
        double ray[3];
        for (int a = 0; a < 3; ++a) ray[a] = c.forward[a] + c.right[a] * sx + c.up[a] * sy;
        const double len = sqrt(ray[0] * ray[0] + ray[1] * ray[1] + ray[2] * ray[2]);
        if (len > 1e-9) {
            for (int a = 0; a < 3; ++a) ray[a] = ray[a] / len;
        } else {
            for (int a = 0; a < 3; ++a) ray[a] = c.forward[a];
        }
        if (ray[1] > 0.0) {
            // the sky image holds the zenith angle as a float
            const float zen = float(acos(fmax(0.0, fmin(1.0, ray[1]))) * 180.0 / kPiD);
            const double wl = double(wavelengths[b]);
            const double wl_nm = (wl > 0.0 && wl <= 50.0) ? wl * 1000.0 : wl;
            v = float(sky_value(wl_nm, double(zen), as_temperature != 0, sky_t));
        }
    }
    image[i] = v;
}

inline unsigned blocks(size_t n, unsigned b) { return unsigned((n + b - 1) / b); }

}  // namespace

namespace {
double hdot(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
double hlen(const double* v) { return std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]); }
void hnormalize(double* v, const double* fallback)
{
    const double n = hlen(v);
    for (int a = 0; a < 3; ++a) v[a] = n > 1e-9 ? v[a] / n : fallback[a];
}
void hcross(const double* a, const double* b, double* r)
{
    const double x = a[1] * b[2] - a[2] * b[1], y = a[2] * b[0] - a[0] * b[2],
                 z = a[0] * b[1] - a[1] * b[0];
    r[0] = x;
    r[1] = y;
    r[2] = z;
}
}  // namespace

Camera camera(const facetcu_sensor& s, double* naming_zenith, double* naming_azimuth)
{
    // server.mjs:1134-1301 in the same operation order
    const double pi = 3.141592653589793;
    Camera c{};
    c.width = s.width ? s.width : 512;
    c.height = s.height ? s.height : 512;
    c.perspective = s.perspective ? 1 : 0;
    c.scene_w = std::max(1e-6, s.scene_x != 0.0 && std::isfinite(s.scene_x) ? s.scene_x : 1.0);
    c.scene_d = std::max(1e-6, s.scene_y != 0.0 && std::isfinite(s.scene_y) ? s.scene_y : 1.0);
    const bool placed = std::isfinite(s.position[0]) && std::isfinite(s.position[1]) &&
                        std::isfinite(s.position[2]);
    const double world[3] = {placed ? s.position[0] : c.scene_w / 2,
                             placed ? s.position[1] : c.scene_d / 2, placed ? s.position[2] : 3000.0};
    c.cam_pos[0] = world[0] - c.scene_w / 2;
    c.cam_pos[1] = std::max(0.01, world[2]);
    c.cam_pos[2] = world[1] - c.scene_d / 2;
    const double z = (std::isfinite(s.view_zenith) ? s.view_zenith : 0.0) * pi / 180;
    const double a = (std::isfinite(s.view_azimuth) ? s.view_azimuth : 0.0) * pi / 180;
    c.out[0] = std::sin(z) * std::cos(a);
    c.out[1] = std::cos(z);
    c.out[2] = std::sin(z) * std::sin(a);
    for (int k = 0; k < 3; ++k) c.forward[k] = -c.out[k];
    // cameraBasis: north-up for a parallel sensor, world-up for a perspective one
    const double north[3] = {1, 0, 0}, world_up[3] = {0, 1, 0};
    const double* preferred = c.perspective ? world_up : north;
    const double* fallback = c.perspective ? north : world_up;
    double up[3];
    const double pp = hdot(preferred, c.forward);
    for (int k = 0; k < 3; ++k) up[k] = preferred[k] - pp * c.forward[k];
    if (hlen(up) <= 1e-9) {
        const double q = hdot(fallback, c.forward);
        for (int k = 0; k < 3; ++k) up[k] = fallback[k] - q * c.forward[k];
    }
    const double fx[3] = {1, 0, 0}, fz[3] = {0, 0, 1};
    hnormalize(up, fx);
    hcross(c.forward, up, c.right);
    hnormalize(c.right, fz);
    double up2[3];
    hcross(c.right, c.forward, up2);
    hnormalize(up2, up);
    for (int k = 0; k < 3; ++k) c.up[k] = up2[k];
    c.tan_half = 1.0;
    if (c.perspective) {
        const double fov = std::max(0.1, std::min(120.0, s.fov != 0.0 && std::isfinite(s.fov) ? s.fov : 60.0));
        c.tan_half = std::tan(fov * 0.5 * pi / 180);
    }
    const double W = c.width, H = c.height, aspect = W / H;
    double mnx, mxx, mny, mxy;
    if (c.perspective) {
        mnx = -1;
        mxx = 1;
        mny = -1;
        mxy = 1;
    } else {
        mnx = INFINITY;
        mxx = -INFINITY;
        mny = INFINITY;
        mxy = -INFINITY;
        const double corners[4][3] = {{-c.scene_w / 2, 0, -c.scene_d / 2},
                                      {-c.scene_w / 2, 0, c.scene_d / 2},
                                      {c.scene_w / 2, 0, -c.scene_d / 2},
                                      {c.scene_w / 2, 0, c.scene_d / 2}};
        for (const auto& p : corners) {
            const double px = hdot(p, c.right), py = hdot(p, c.up);
            mnx = std::min(mnx, px);
            mxx = std::max(mxx, px);
            mny = std::min(mny, py);
            mxy = std::max(mxy, py);
        }
    }
    double rx = std::max(1e-6, mxx - mnx), ry = std::max(1e-6, mxy - mny);
    const double cx = (mnx + mxx) / 2, cy = (mny + mxy) / 2;
    if (rx / ry > aspect)
        ry = rx / aspect;
    else
        rx = ry * aspect;
    rx *= 1 + 0.5 / W;
    ry *= 1 + 0.5 / H;
    c.range_x = rx;
    c.range_y = ry;
    c.min_x = cx - rx / 2;
    c.max_y = cy + ry / 2;
    double east = c.scene_d, northr = c.scene_w;
    if (east / northr > aspect)
        northr = east / aspect;
    else
        east = northr * aspect;
    c.orth_east = east / 1.0;
    c.orth_north = northr / 1.0;
    c.orth_min_z = -c.orth_east / 2;
    c.orth_max_x = c.orth_north / 2;
    if (naming_zenith && naming_azimuth) {
        if (c.perspective) {
            const double h = std::hypot(c.out[0], c.out[2]);
            *naming_zenith = std::acos(std::max(-1.0, std::min(1.0, c.out[1]))) * 180 / pi;
            *naming_azimuth =
                h < 1e-9 ? 0.0 : std::fmod(std::atan2(c.out[2], c.out[0]) * 180 / pi + 360, 360.0);
        } else {
            *naming_zenith = s.view_zenith;
            *naming_azimuth = s.view_azimuth;
        }
    }
    return c;
}

void render(const Camera& c, uint32_t F, const facetcu_vertex* V, const float* values,
            uint32_t nb, size_t S, const float* wavelengths, bool as_temperature, double sky_t,
            Scratch& w, float* image, int32_t* sides, uint32_t* counts, cudaStream_t s)
{
    const size_t n = size_t(c.width) * c.height;
    FCU_CHECK(cudaMemsetAsync(counts, 0, 3 * sizeof(uint32_t), s));
    FCU_CHECK(cudaMemsetAsync(w.zbuf, 0, n * sizeof(ulonglong2), s));
    if (F) {
        // A warp takes as many facets as share some 512 of the image's pixels, fewer
        // lanes than that do the projection's doubles (a warp of them costs the same)
        // for nothing, more leave too long a queue of boxes; and no more than leave
        // 16 warps an SM, unless the image is small.  Side images in us with 32 facets
        // a warp / 2, 4 and 16 warps an SM: 2,000 facets on 64 x 64 57 / 57, 69, 81 (a
        // warp per facet of old: 86), 4,000 on 1,024 x 1,024 2,751 / 917, 743, 659
        // (1,547), 30,000 1,605 / 1,654, 1,655, 1,498 (2,522).
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const uint32_t spread = F / (16u * uint32_t(std::max(sms, 1)));
        const uint32_t of_image = uint32_t(std::min<size_t>(512 * size_t(F) / n, 32u));
        const uint32_t per_warp = std::clamp(std::max(spread, of_image), 1u, 32u);
        k_raster<<<blocks(F, per_warp * kRasterThreads / 32), kRasterThreads, 0, s>>>(
            F, per_warp, V, c, w.zbuf, w.side, w.large, counts + 2);
        FCU_LAUNCH("k_raster");
        k_raster_large<<<8u * uint32_t(std::max(sms, 1)), 256, 0, s>>>(V, c, w.zbuf, w.large,
                                                                      counts + 2);
        FCU_LAUNCH("k_raster_large");
    }
    k_observed<<<blocks(n, 256), 256, 0, s>>>(n, w.zbuf, w.side, w.index, counts);
    FCU_LAUNCH("k_observed");
    int32_t* out = w.index;
    if (!c.perspective) {
        k_nadir<<<blocks(c.width, 32) * blocks(c.height, 8), 256, 0, s>>>(c, w.index, sides,
                                                                          counts + 1);
        FCU_LAUNCH("k_nadir");
        out = sides;
    } else {
        FCU_CHECK(cudaMemcpyAsync(sides, w.index, n * 4, cudaMemcpyDeviceToDevice, s));
        FCU_CHECK(cudaMemcpyAsync(counts + 1, counts, 4, cudaMemcpyDeviceToDevice, s));
        out = sides;
    }
    if (nb) {
        k_fill<<<blocks(n * nb, 256), 256, 0, s>>>(c, nb, S, out, values, wavelengths,
                                                   as_temperature ? 1 : 0, sky_t, image);
        FCU_LAUNCH("k_fill");
    }
}

}  // namespace image
}  // namespace facetcu
