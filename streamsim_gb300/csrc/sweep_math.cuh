// sweep_math.cuh — the stop test shared by the batched solver's sweeps.
#pragma once
#include <cstdint>

namespace facetcu {

constexpr int kMaxP = 128;  // columns of the widest panel; the statistics' stride

// The per-side stop test: |dB_s| / max(|B_s|, kSideFloor * max|B|) <= tol
// per column, the form of the accuracy bar (relative error per side, with
// sides below 1e-6 of the column's maximum measured against that floor).
constexpr float kSideFloor = 1e-6f;
__device__ __forceinline__ float rel_change(float d, float b, float floor_abs)
{
    d = fabsf(d);
    if (d == 0.0f) return 0.0f;
    const float den = fmaxf(fabsf(b), floor_abs);
    return den > 0.0f ? d / den : INFINITY;
}

}  // namespace facetcu
