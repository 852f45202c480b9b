// Shared-memory Stockham FFT building blocks for sm_103a.
//
// A CTA holds B transforms of N points each in shared memory (complex64,
// padded layout).  Each transform is worked by T = N/8 threads that each keep
// 8 points in registers per stage: radix-8 stages, then one radix-4 or
// radix-2 stage for sizes that are not a power of 8.  Stage s with span Ns
// reads point b + k*N/R, twiddles it by W_{Ns*R}^{(b mod Ns) k}, runs an R-point
// DFT and writes point (b/Ns)*Ns*R + (b mod Ns) + m*Ns (autosort: natural
// order in, natural order out, no bit reversal).
//
// Layout: logical point i of a transform lives at pad_idx(i) = i + i/16, one
// spare complex every 16, which spreads the stride-R stores of the early
// stages over all banks; transforms are tstride(N) (odd) complexes apart.
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

__host__ __device__ constexpr int pad_idx(int i) { return i + (i >> 4); }
__host__ __device__ constexpr int padded_len(int n) { return n + (n >> 4); }
// Distance between consecutive transforms of a CTA in shared memory: odd, so
// that B transforms read at the same logical index fall in distinct banks.
__host__ __device__ constexpr int tstride(int n) { return padded_len(n) + 1; }
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
// packed.  (600 x 1024^2 to 512^3 3398 us, with packed first sums 3399.  The
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

// One Stockham stage on a transform held in shared memory (in place).
// Every thread of the CTA must call it (it contains __syncthreads()); threads
// with active == false only take part in the barriers.
template <int N, int R, int NS, int DIR>
__device__ __forceinline__ void fft_stage(float2* s, int j, const float2* __restrict__ tw, bool active) {
    constexpr int T = N / 8;
    constexpr int NB = 8 / R;
    float2 x[8];
    if (active) {
#pragma unroll
        for (int t = 0; t < NB; ++t) {
            const int b = j + t * T;
#pragma unroll
            for (int k = 0; k < R; ++k) x[t * R + k] = s[pad_idx(b + k * (N / R))];
        }
    }
    __syncthreads();
    if (active) {
#pragma unroll
        for (int t = 0; t < NB; ++t) {
            const int b = j + t * T;
            const int p = b % NS;
            if constexpr (NS > 1) {
#pragma unroll
                for (int k = 1; k < R; ++k) {
                    float2 w = __ldg(&tw[p * k * (kTwN / (NS * R))]);
                    if constexpr (DIR > 0) w.y = -w.y;
                    x[t * R + k] = c_mul(x[t * R + k], w);
                }
            }
            if constexpr (R == 8) dft8<DIR>(&x[t * R]);
            else if constexpr (R == 4) dft4<DIR>(x[t * R], x[t * R + 1], x[t * R + 2], x[t * R + 3]);
            else dft2<DIR>(x[t * R], x[t * R + 1]);
            const int base = (b / NS) * NS * R + p;
#pragma unroll
            for (int m = 0; m < R; ++m) s[pad_idx(base + m * NS)] = x[t * R + m];
        }
    }
    __syncthreads();
}

// Full N-point transform of the padded shared-memory array s, worked by
// thread j in [0, N/8) of the transform.  Input and output in natural order.
template <int N, int DIR>
__device__ __forceinline__ void fft_smem(float2* s, int j, const float2* __restrict__ tw, bool active = true) {
    static_assert(N >= 64 && N <= kTwN && (N & (N - 1)) == 0, "power-of-two size in [64, 4096]");
    constexpr int L2 = ilog2c(N);
    constexpr int n8 = L2 / 3;
    constexpr int rem = L2 % 3;
    fft_stage<N, 8, 1, DIR>(s, j, tw, active);
    fft_stage<N, 8, 8, DIR>(s, j, tw, active);
    if constexpr (n8 >= 3) fft_stage<N, 8, 64, DIR>(s, j, tw, active);
    if constexpr (n8 >= 4) fft_stage<N, 8, 512, DIR>(s, j, tw, active);
    constexpr int NSf = 1 << (3 * n8);
    if constexpr (rem == 1) fft_stage<N, 2, NSf, DIR>(s, j, tw, active);
    if constexpr (rem == 2) fft_stage<N, 4, NSf, DIR>(s, j, tw, active);
}

}  // namespace tdm
