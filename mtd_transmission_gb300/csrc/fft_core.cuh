// Complex arithmetic and register butterflies of the FFT passes for sm_103a, and
// the sizes of their twiddle table.
//
// Sign conventions follow FFTW: DIR = -1 is exp(-2 pi i jk/N) (forward),
// DIR = +1 is exp(+2 pi i jk/N) (backward); neither is normalised.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace tdm {

constexpr int kTwN = 4096;  // twiddle table size: exp(-2 pi i k / 4096)

// Points per lane of the warp-resident FFT of size n (fft_warp.cuh).
__host__ __device__ constexpr int warp_fft_e(int n) { return n >= 2048 ? 64 : n >= 512 ? 32 : n >= 128 ? 16 : 8; }
// Offset of the per-lane twiddle factors of the n-point warp FFT in the
// device twiddle table (after the kTwN-entry table): one n-entry block per
// size 64, 128, ..., 2048.
__host__ __device__ constexpr int twr_offset(int n) { return kTwN + n - 64; }
constexpr int kTwTotal = kTwN + 4096 - 64;

__host__ __device__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n >> 1); }

// A complex value is a register pair, and the packed FP32 instructions of this
// GPU work on both halves at once: an addition, a real scaling or a butterfly
// with a common real factor is one instruction instead of two.  (A product
// with a complex factor or +-i would need the halves swapped by moves first, so
// those stay scalar.)  The FFT passes issue two thirds of their instructions
// for arithmetic: extraction of 400 x 1024^2 row pass 512 -> 478 us, column pass
// 280 -> 262 us, a 600 x 1024^2 volume 4.02 -> 3.90 ms.
__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) {
    float2 r;
    asm("sub.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return r;
}
__device__ __forceinline__ float2 c_mul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 c_scale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
__device__ __forceinline__ float2 c_conj(float2 a) { return make_float2(a.x, -a.y); }

// A value of the cap transforms.  The compiler may fuse a product (by the window,
// by 1/sqrt 2) into the scalar addition that follows, but not into a packed one,
// and the caps keep that rounding: the support mask marks the cells whose real
// part is not exactly 0, a transform's value is 0 by accident in 1 of 1e8 cells,
// and after any change of rounding in other cells.  So the first sums of a
// butterfly, the only ones that products reach, are scalar for this type; the rest is
// packed.  Which of them the compiler fuses is its own choice (nvcc 13.0, -fmad on), so
// another compiler may set such a cell's mark differently.  (600 x 1024^2 to 512^3 3398 us, with packed first sums 3399.  The
// mixed-radix butterflies take their products through fma() or shared memory and
// need no such type; all scalar they took 500 x 250^2 to 512^3 from 1450 to 1555 us.)
struct alignas(8) Fusable {
    float x, y;
    Fusable() = default;
    __device__ __forceinline__ Fusable(float2 v) : x(v.x), y(v.y) {}
    __device__ __forceinline__ operator float2() const { return make_float2(x, y); }
};
__device__ __forceinline__ float2 c_add(Fusable a, Fusable b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(Fusable a, Fusable b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ Fusable c_scale(Fusable a, float s) { return make_float2(a.x * s, a.y * s); }

// a * (DIR * i)
template <int DIR>
__device__ __forceinline__ float2 mul_dir_i(float2 a) {
    return DIR < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}

template <int DIR>
__device__ __forceinline__ void dft2(float2& a0, float2& a1) {
    float2 t = a0;
    a0 = c_add(t, a1);
    a1 = c_sub(t, a1);
}

template <int DIR, class V>
__device__ __forceinline__ void dft4(V& a0, V& a1, V& a2, V& a3) {
    const float2 t0 = c_add(a0, a2), t1 = c_sub(a0, a2);
    const float2 t2 = c_add(a1, a3), d = c_sub(a1, a3);
    a0 = c_add(t0, t2);
    a2 = c_sub(t0, t2);
    a1 = make_float2(t1.x - DIR * d.y, t1.y + DIR * d.x);  // t1 + DIR i d
    a3 = make_float2(t1.x + DIR * d.y, t1.y - DIR * d.x);
}

template <int DIR, class V>
__device__ __forceinline__ void dft8(V* x) {
    V e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6];
    V o0 = x[1], o1 = x[3], o2 = x[5], o3 = x[7];
    dft4<DIR>(e0, e1, e2, e3);
    dft4<DIR>(o0, o1, o2, o3);
    const float r = 0.70710678118654752440f;
    const float2 rp = make_float2(r, r), rm = make_float2(-r, -r);
    // o1 *= exp(DIR i pi/4) = r u1, o2 *= DIR i, o3 *= exp(DIR 3 i pi/4) = r u3
    const float2 u1 = make_float2(o1.x - DIR * o1.y, DIR * o1.x + o1.y);
    const float2 u3 = make_float2(-o3.x - DIR * o3.y, DIR * o3.x - o3.y);
    x[0] = c_add(float2(e0), float2(o0));
    x[4] = c_sub(float2(e0), float2(o0));
    x[1] = __ffma2_rn(rp, u1, e1);
    x[5] = __ffma2_rn(rm, u1, e1);
    x[2] = make_float2(e2.x - DIR * o2.y, e2.y + DIR * o2.x);
    x[6] = make_float2(e2.x + DIR * o2.y, e2.y - DIR * o2.x);
    x[3] = __ffma2_rn(rp, u3, e3);
    x[7] = __ffma2_rn(rm, u3, e3);
}

}  // namespace tdm
