// diffuse_mean (compensated.cuh) on the CPU: the float it returns against the
// long double value of (skyc L + s + c) / d, in units of the result's last place,
// beside the float of the same quotient in doubles.  Prints one line per range:
// name, worst error of the pair form, of the double form, times they differ.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

#define __device__
#define __forceinline__ inline
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline uint32_t max(uint32_t a, uint32_t b) { return a > b ? a : b; }
#include "../../streamsim_gb300/csrc/compensated.cuh"

static double error_of(float got, long double want)
{
    if (std::isnan(got)) return std::isnan(want) ? 0.0 : INFINITY;
    const float w = float(want);
    if (std::isinf(got) || std::isinf(w)) return got == w ? 0.0 : INFINITY;
    const float a = std::max(std::fabs(w), 1.17549435e-38f);
    const long double ulp = (long double)std::nextafter(a, INFINITY) - (long double)a;
    return double(std::fabs((long double)got - want) / ulp);
}

int main()
{
    std::mt19937_64 g(12345);
    auto uniform = [&](double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(g); };
    struct Range {
        const char* name;
        double lo, hi;      // decimal exponent of the radiosities
        uint32_t most;      // terms
        uint32_t count;     // largest count of a term
        double sky;         // exponent of the sky radiance (NAN: 0)
    };
    const Range ranges[] = {
        {"radiation", -2, 3, 400, 64, 2},     {"bright", 3, 12, 400, 64, 4},
        {"dim", -12, -2, 400, 64, -3},        {"no_sky", -2, 3, 400, 64, NAN},
        {"few", -2, 3, 3, 64, 2},             {"large_counts", -2, 3, 100, 1u << 20, 2},
        {"tiny", -37, -20, 100, 64, -30},     {"tiniest", -44, -36, 20, 8, -40},
        {"huge", 30, 36, 4, 64, 30},          {"mixed", -30, 30, 50, 64, 2},
    };
    for (const Range& r : ranges) {
        double pair = 0.0, plain = 0.0;
        long differ = 0;
        for (int k = 0; k < 100000; ++k) {
            facetcu::Csum a{0.0f, 0.0f};
            const uint32_t n = uint32_t(uniform(0, r.most + 1));
            uint64_t d = 0;
            for (uint32_t i = 0; i < n; ++i) {
                const uint32_t c = 1u + uint32_t(uniform(0, r.count));
                const float v = uniform(0, 1) < 0.05 ? 0.0f : float(std::pow(10.0, uniform(r.lo, r.hi)));
                facetcu::csum_term(a, c, v);
                d += c;
            }
            const uint32_t skyc = uint32_t(uniform(0, 200));
            d = std::min<uint64_t>(d + skyc, 0xffffffffu);
            if (d == 0) continue;
            const float L = std::isnan(r.sky) ? 0.0f : float(std::pow(10.0, r.sky) * uniform(0.1, 10));
            const long double want = ((long double)skyc * L + (long double)a.s + (long double)a.c) /
                                     (long double)d;
            const float got = facetcu::diffuse_mean(a, skyc, L, uint32_t(d));
            const float old = float((double(skyc) * double(L) + facetcu::csum_value(a)) / double(d));
            pair = std::max(pair, error_of(got, want));
            plain = std::max(plain, error_of(old, want));
            differ += got != old && !(std::isnan(got) && std::isnan(old));
        }
        std::printf("%s %.6f %.6f %ld\n", r.name, pair, plain, differ);
    }
    // what is not a number or not finite comes out as in doubles
    const float odd[] = {0.0f, -0.0f, 1.0f, 3.0e38f, 1.0e-45f, INFINITY, -INFINITY, NAN, -1.0f, -3.0e38f};
    long wrong = 0;
    for (float s : odd)
        for (float c : odd)
            for (float L : odd)
                for (uint32_t skyc : {0u, 7u, 0xffffffffu})
                    for (uint32_t d : {1u, 300u, 0xffffffffu}) {
                        const facetcu::Csum a{s, std::fabs(c) > 1.0f ? 0.0f : c * 1e-8f};
                        const float got = facetcu::diffuse_mean(a, skyc, L, d);
                        const float old = float((double(skyc) * double(L) + facetcu::csum_value(a)) / double(d));
                        const bool same = got == old || (std::isnan(got) && std::isnan(old)) ||
                                          (std::isfinite(old) && std::isfinite(got) &&
                                           std::fabs(got - old) <= 1.2e-7f * std::fabs(old) + 1.0e-44f);
                        if (!same && wrong++ < 6)
                            std::printf("# s %g c %g L %g skyc %u d %u: %g, in doubles %g\n", a.s, a.c, L, skyc, d, got, old);
                    }
    std::printf("odd %ld 0 0\n", wrong);
    return 0;
}
