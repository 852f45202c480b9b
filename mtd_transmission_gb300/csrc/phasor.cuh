// Field values as amplitude and unit phasor, and the phasor's gradient: shared by
// the field and Volkov passes of both FFT engines (k_fields.cu, k_generic.cu).
#pragma once

#include "quotient.cuh"
#include "tdm_internal.cuh"

namespace tdm {

constexpr float kInvTwoPi = 0.15915494309189535f;

// Amplitude |u| and unit phasor u/|u| (1 where u = 0: atan2(0, 0) = 0) from one
// reciprocal square root r: |u|^2 r, corrected by one step of Newton's iteration
// for the square root, and u r.  A field value whose square leaves the normal range
// is scaled first, and its amplitude is hypotf's.
__device__ __forceinline__ float amplitude(float2 u, float2& z) {
    auto unit = [&](float2 w) {
        const float m2 = fmaf(w.x, w.x, w.y * w.y), r = rsqrtf(m2), m = m2 * r;
        z = make_float2(w.x * r, w.y * r);
        return fmaf(fmaf(-m, m, m2), 0.5f * r, m);
    };
    const float m2 = fmaf(u.x, u.x, u.y * u.y);
    if (m2 > 1e-30f && m2 < 1e30f) return unit(u);
    const float m = hypotf(u.x, u.y);
    if (m > 0.0f && m < __int_as_float(0x7f800000)) {
        const float k = m < 1.0f ? 0x1p100f : 0x1p-100f;
        unit(make_float2(u.x * k, u.y * k));
    } else {
        z = m == 0.0f ? make_float2(1.0f, 0.0f) : make_float2(u.x / m, u.y / m);
    }
    return m;
}

// What the column pass leaves per field pixel.  FIELD (C_ABER off): the field
// itself is the result.  The rest leave the amplitude and, for Volkov, the unit
// phasor; for Herraez or no unwrapping, the wrapped phase.  Volkov's solve
// gives the unwrapped phase less the wrapped phase's mean, a constant that the
// aberration fit's constant term takes out of the field, so the phase is formed
// only where the unwrapped phase itself is wanted (VOLKOV_PHASE), with each CTA's
// sum of it in psum[a * kPhaseParts + blockIdx.x] (FP32 per thread and warp, FP64
// across the warps in a fixed order).
enum FieldMode { FIELD, PHASE, VOLKOV, VOLKOV_PHASE };

// Re(-i g / Z) / 2pi for a unit phasor Z: g conj(Z) / |Z|^2, where |Z|^2 = 1 + d
// with d a few roundings, so 1 / |Z|^2 is 2 - |Z|^2 to d^2 (the division took a
// fifth of the row pass: 100 angles of 256^2 32 -> 27 us).
__device__ __forceinline__ float phasor_gradient(float2 g, float2 z) {
    return (g.y * z.x - g.x * z.y) * (2.0f - fmaf(z.x, z.x, z.y * z.y)) * kInvTwoPi;
}

}  // namespace tdm
