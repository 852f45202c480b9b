// Ewald-cap geometry of retroPropag_Born (Reconstruction/src/fonctions.cpp:875-935),
// shared by the cap passes for every field size and by the forward
// operator's sampling.
#pragma once

#include "tdm_internal.cuh"

namespace tdm {

// v mod F for v in [0, 2F) (a bin plus a specular coordinate).
__device__ __forceinline__ int wrap_f(int v, int F) { return v >= F ? v - F : v; }

// fzm0 of an angle (fonctions.cpp:893-899): in FP64, and as a pair of floats
// whose sum it is to about 2^-48; f is negative when the angle is skipped.  It is
// the height sqrt(rayon^2 - fd^2) at the specular position, so the tables of
// cap heights have it for every position in the field (an FP64 square root by
// one thread of each CTA kept the others waiting for a few thousand cycles); a
// position from outside is computed.
struct CapFz {
    double d;
    float f, lo;
};
static __device__ __noinline__ double cap_fzm0_outside(const Params& p, int2 ps) {
    const int fxm0 = ps.x - p.N, fym0 = ps.y - p.N;
    const double c = p.rayon * p.rayon - fxm0 * fxm0 - fym0 * fym0;
    return (round(c) >= 0) ? sqrt(c) : -1.0;
}
__device__ __forceinline__ CapFz cap_fzm0(const Params& p, int2 ps, const double* __restrict__ s_tab,
                                          const float2* __restrict__ s_pair) {
    CapFz fz;
    if ((unsigned)ps.x < (unsigned)p.F && (unsigned)ps.y < (unsigned)p.F) {
        const float2 t = s_pair[ps.y * p.F + ps.x];
        fz = CapFz{s_tab[ps.y * p.F + ps.x], t.x, t.y};
    } else {
        fz.d = cap_fzm0_outside(p, ps);
        fz.f = (float)fz.d;
        fz.lo = (float)(fz.d - (double)fz.f);
    }
    if (!(fz.f >= 0.0f)) fz.f = -1.0f;  // NaN below the sphere
    return fz;
}

// Plane z of the cap cell of FFT bin (kx, ky) of an angle with specular
// position ps and height fz: round(sqrt(fdz^2) - fzm0) in FP64
// (fonctions.cpp:903-921), or -1 outside the NA disc or for a skipped angle; *sf
// is sqrt(r^2 - fd^2) in float for the cell's weight.  A plane outside the cap
// band sets *err and gives -1.  FP64 instructions run at 1/64 of the FP32 rate on
// this GPU, so the decision is taken in FP32 where that is certain: by the
// float heights unless they come within 1e-3 of a rounding boundary (one bin in
// 500, but one warp in 15), then by the heights as pairs of floats, whose
// difference is right to 1e-10, unless that comes within 1e-8.  With FP64 as the
// first fallback its pipe bounded the column pass: 100 angles of 256^2 58 us.
__device__ __forceinline__ int cap_plane(const Params& p, int2 ps, CapFz fz, int kx, int ky,
                                         const double* __restrict__ s_tab, const float2* __restrict__ s_pair,
                                         float* sf, int* __restrict__ err) {
    const int F = p.F, N = p.N;
    const int fdx = wrap_f(kx + ps.x, F) - N, fdy = wrap_f(ky + ps.y, F) - N;
    if (!(fz.f >= 0.0f) || fdx * fdx + fdy * fdy >= p.disc_thr) return -1;  // fz is sqrt(c) >= 0 or -1
    const int ti = (fdy + N) * F + fdx + N;
    // sqrt(r^2 - fd^2) in float: computed from the exact integer when r^2 < 2^24 (equal to the table)
    *sf = p.r2i ? __fsqrt_rn((float)(p.r2i - fdx * fdx - fdy * fdy)) : s_pair[ti].x;
    const float d = *sf - fz.f, below = floorf(d), edge = below + 0.5f;
    const float fr = d - below;
    float koz;
    if (fabsf(fr - 0.5f) > 1e-3f) {
        koz = floorf(d + 0.5f);
    } else {
        const float v = d - *sf, e = (*sf - (d - v)) - (fz.f + v);  // d + e = *sf - fz.f exactly
        const float t = (d - edge) + (e + (s_pair[ti].y - fz.lo));
        koz = fabsf(t) > 1e-8f ? (t > 0.0f ? below + 1.0f : below) : (float)round(s_tab[ti] - fz.d);
    }
    const int z = (int)koz + p.D / 2;
    if (z < p.zmin || z >= p.zmin + p.band) {
        if (err) atomicOr(err, 1);
        return -1;
    }
    return z;
}

// Cap-cell weight (k0/pi)(-2pi) sdz dx^2 (-1)^(kx+ky) of retroPropag_Born
// (fonctions.cpp:902,927) with the recentring sign of the per-field spectrum.
// ir = (float)p.inv_rayon, converted once by the caller.
__device__ __forceinline__ float cap_weight(const Params& p, float sf, float ir, int kx, int ky) {
    const float sg = ((kx + ky) & 1) ? -p.dx2 : p.dx2;
    return p.cap_scale * (sf * ir) * sg;
}

// Voxel column of FFT bin kx of an angle with specular coordinate q (x or y):
// D/2 + fd + N - q, the inverse of the gather's bin (X - D/2) mod F.
__device__ __forceinline__ int cap_col(const Params& p, int k, int q) {
    return p.D / 2 + wrap_f(k + q, p.F) - q;
}

}  // namespace tdm
