// Check of the shortened divisions and square roots of csrc/quotient.cuh and
// csrc/phasor.cuh on the GPU, over random values of the ranges they are used in,
// against CUDA's own division and against 64-bit arithmetic.  Prints one line per
// function: its name, the worst error in units of its bound, and the violations.
#include <cstdio>
#include <cstring>

#include "phasor.cuh"

using namespace tdm;

enum { OVER, OVER_SMALL, OVER_SPECIAL, QUOTIENT, AMPLITUDE, AMPLITUDE_SCALED, PHASOR, GRADIENT, SPECIAL, COUNT };
struct Result {
    unsigned long long bad[COUNT], seen[COUNT];
    float worst[COUNT];
};

__device__ unsigned long long mix(unsigned long long z) {  // splitmix64 (Steele, Lea, Flood 2014)
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ float uniform(unsigned long long h) { return (float)(h >> 40) * 0x1p-24f; }
// mantissa in [1, 2), exponent in [lo, hi], either sign
__device__ float spread(unsigned long long h, int lo, int hi) {
    const float m = 1.0f + (float)(h & 0x7FFFFF) * 0x1p-23f;
    const int e = lo + (int)((h >> 24) % (unsigned)(hi - lo + 1));
    return ldexpf((h >> 63) ? -m : m, e);
}

__device__ void note(Result* r, int id, double error, double bound) {
    atomicAdd(&r->seen[id], 1ull);
    const double q = error / bound;
    if (!(q <= 1.0)) atomicAdd(&r->bad[id], 1ull);
    atomicMax(reinterpret_cast<int*>(&r->worst[id]), __float_as_int((float)q));  // not negative: ordered as integers
}
__device__ bool same(float a, float b) { return a == b || (a != a && b != b); }

__global__ void check(Result* r, int per, float inf) {
    const unsigned long long id = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    for (int i = 0; i < per; ++i) {
        const unsigned long long h = mix(id * per + i), h2 = mix(h), h3 = mix(h2), h4 = mix(h3);
        // a cell's sum over its hit count
        const float n = (float)(1 + (h2 >> 8) % (i & 1 ? 600u : 65535u)), rn = __frcp_rn(n);
        const float x = spread(h, -100, 120);
        note(r, OVER, fabsf(over(x, n, rn) - x / n), 1e-300);  // equal
        const float xs = spread(h, -149, -120);
        note(r, OVER_SMALL, fabsf(over(xs, n, rn) - xs / n), 0x1p-149);
        const float sp[4] = {inf, -inf, inf - inf, 0.0f};
        for (int k = 0; k < 4; ++k) note(r, OVER_SPECIAL, same(over(sp[k], n, rn), sp[k] / n) ? 0.0 : 2.0, 1.0);
        // the Poisson quotient: y = kx^2 + ky^2 of a quadrant of at most 512^2
        const float kx = (float)(h3 % 512) / 1024.0f, ky = (float)((h3 >> 20) % 512) / 1024.0f;
        const float y = kx * kx + ky * ky;
        if (y > 0.0f) {
            const float xq = spread(h4, -60, 60), e = xq / y;
            note(r, QUOTIENT, fabsf(quotient(xq, y) - e), 0x1p-23 * fabs((double)e));  // at most one unit
        }
        // amplitude and unit phasor; |u|^2 has at most 2 roundings of 2^-24, its root half of them, the
        // corrected root one more; the phasor one reciprocal root of 2 units (2^-23) and one rounding more
        for (int big = 0; big < 2; ++big) {
            const float a = big ? spread(h2, -140, 120) : spread(h2, -40, 40);
            const float th = 6.2831853f * uniform(h3);
            const float2 u = make_float2(a * cosf(th), a * sinf(th));
            float2 z;
            const float m = amplitude(u, z);
            const double m64 = sqrt((double)u.x * u.x + (double)u.y * u.y);
            if (!(m64 > 0.0)) continue;
            // (hypotf: at most 3 units, or one unit of 2^-149)
            note(r, big ? AMPLITUDE_SCALED : AMPLITUDE, fabs((double)m - m64),
                 big ? fmax(4 * 0x1p-23 * m64, 0x1p-148) : 3 * 0x1p-24 * m64);
            const double ex = u.x / m64, ey = u.y / m64;
            note(r, PHASOR, sqrt((z.x - ex) * (z.x - ex) + (z.y - ey) * (z.y - ey)), 7 * 0x1p-24);
            // Re(-i g / Z) / 2 pi: the numerator's two products and their difference, 2 - |Z|^2, two products
            const float2 g = make_float2(spread(h4, -10, 10), spread(mix(h4), -10, 10));
            const double zz = (double)z.x * z.x + (double)z.y * z.y;
            const double want = ((double)g.y * z.x - (double)g.x * z.y) / zz * 0.15915494309189533577;
            const double gm = sqrt((double)g.x * g.x + (double)g.y * g.y) * 0.15915494309189533577;
            note(r, GRADIENT, fabs((double)phasor_gradient(g, z) - want), 8 * 0x1p-24 * gm);
        }
    }
    if (id == 0) {
        float2 z;
        float m = amplitude(make_float2(0.0f, 0.0f), z);
        note(r, SPECIAL, m == 0.0f && z.x == 1.0f && z.y == 0.0f ? 0.0 : 2.0, 1.0);
        m = amplitude(make_float2(inf, 1.0f), z);
        note(r, SPECIAL, m == inf ? 0.0 : 2.0, 1.0);
        m = amplitude(make_float2(inf - inf, 1.0f), z);
        note(r, SPECIAL, m != m ? 0.0 : 2.0, 1.0);
        m = amplitude(make_float2(3e38f, 0.0f), z);
        note(r, SPECIAL, fabs(m / 3e38 - 1) < 1e-6 && fabsf(z.x - 1.0f) < 1e-6f && z.y == 0.0f ? 0.0 : 2.0, 1.0);
        m = amplitude(make_float2(0.0f, 0x1p-149f), z);
        note(r, SPECIAL, m == 0x1p-149f && z.x == 0.0f && fabsf(z.y - 1.0f) < 1e-6f ? 0.0 : 2.0, 1.0);
    }
}

int main() {
    Result *d = nullptr, h;
    if (cudaMalloc(&d, sizeof(Result)) || cudaMemset(d, 0, sizeof(Result))) return 2;
    check<<<256, 256>>>(d, 64, __builtin_inff());
    if (cudaMemcpy(&h, d, sizeof(Result), cudaMemcpyDeviceToHost)) return 2;
    cudaFree(d);
    const char* names[COUNT] = {"over", "over_small", "over_special", "quotient", "amplitude", "amplitude_scaled",
                                "phasor", "gradient", "special"};
    for (int i = 0; i < COUNT; ++i) std::printf("%s %.3g %llu %llu\n", names[i], h.worst[i], h.bad[i], h.seen[i]);
    return 0;
}
