// Off-axis extraction kernels (holo2TF_UBorn, pretraitement_hors_axe_CPU/fonctions.cpp:279-304),
// shared by the context entry points (k_extract.cu) and the allocation-free
// entry point (tdm_noalloc.cu).  See k_extract.cu for the algorithm.
#pragma once

#include "tdm_internal.cuh"
#include "fft_warp.cuh"
#include "bulk_copy.cuh"

namespace tdm {
namespace extract {

// The row pass runs in CTAs of 8 warps, a warp per G row pairs: it packs two
// real rows into one complex transform and keeps the crop's kx band, written row
// by row (inter[a][y][c]).  The column pass's lanes run across columns (ColFFT):
// it reads the band's rows, transforms the columns in registers and stores the
// crop's rows (to the caller's buffer as well, on request), with the crop's
// partial specular-peak winners on request (one record per warp), so that neither pass stages its data for the other's order.
// Bound by issue (the row pass 63 % active at two CTAs an SM).  400 x 1024^2, F =
// 256: rows 479 us with the band stored column by column through a tile, 397 like
// this; columns 270 us as a warp per stored column with the crop through a tile,
// 294 like this (64-byte pieces instead of whole columns, but 16 columns a CTA
// leave one CTA an SM: 349); 64 x 2048^2 422 + 222 us, now 349 + 224.
template <int H>
struct ExtractCfg {
    using W = WarpFFT<H>;
    static constexpr int NT = 256;         // threads per CTA (rows pass)
    static constexpr int P = 8 * W::G;     // row pairs per CTA (rows pass)
    // columns per CTA: from 32 lanes a transform on 8, so that two CTAs (H =
    // 1024) fit an SM's registers
    using Cols = ColFFT<H, (W::T >= 32 ? 8 : 16)>;
    // row-pass CTAs per SM that the registers are capped for (shared memory
    // would allow 3 up to H = 1024, but capping to 80 registers for them
    // spills and measured slower than 2)
    static constexpr int ROWS_CTAS = H >= 2048 ? 1 : 2;
    static constexpr int COLS_CTAS = Cols::NT >= 512 || H >= 2048 ? 1 : 512 / Cols::NT;
    static constexpr size_t SMEM_ROWS = (size_t)P * W::STRIDE * sizeof(float2);
    static dim3 grid_rows(int m) { return dim3(H / (2 * P), m); }
    static dim3 grid_cols(int F, int m) { return dim3((F + Cols::B - 1) / Cols::B, m); }
    static int arg_parts(int F) { return (int)grid_cols(F, 1).x * (Cols::NT / 32); }
};

// Lanes' elements n1 whose pixels x = j + T n1 can fall in the hologram
// window's tapers: the first and the last win_edge of the E.  The window
// (Tukey, alpha 0.05) is exactly 1 on the others; window_edge_ok checks that
// on the host before a launch.
template <int H>
constexpr int win_edge() { return H >= 2048 ? 2 : 1; }
inline bool window_edge_ok(int H, int2 flat, int edge) {
    const int T = H / warp_fft_e(H);
    return flat.x <= T * edge && flat.y >= H - T * edge - 1;
}

// Row pass.  win[x] = ((-1)^x w(x), -2^23 (-1)^x w(x)) is the hologram window
// with the sign modulation of the first fftshift (hologram_window): a pixel p
// is read as the float m = 2^23 + p (its bits OR 0x4B000000) and fma(m, ws,
// cs) is p (-1)^x w(x) rounded once, with no integer-to-float conversion.  On
// the window's flat middle (-1)^x = (-1)^j, so the lane's own (+-1, -+2^23)
// stands for the table there.  The rows' factors (-1)^y w(y) are applied when
// the two packed rows are separated.  ref_inv (may be null) is the H x H
// reciprocal of the reference amplitude, applied to every pixel
// (main.cpp:147).  BULK: each warp's 2G rows (its G row pairs, consecutive in
// memory) are staged in shared memory by one bulk copy and read from there;
// requires a 16-byte aligned stack.  Otherwise the lanes load the pixels
// directly.  A bulk copy that does not complete within wait_polls polls sets
// bit 1 of *err (the call then fails); the warp then waits for its copy again,
// up to the full bound kMbarPolls, so that no copy is left in flight into the
// shared memory of a finished CTA.
template <int H, bool BULK>
__global__ void __launch_bounds__(ExtractCfg<H>::NT, ExtractCfg<H>::ROWS_CTAS)
k_extract_rows(const void* __restrict__ holos, int bits, const float2* __restrict__ win,
               const float* __restrict__ ref_inv, const float2* __restrict__ tw, float2* __restrict__ inter, int F,
               int x0, int* __restrict__ err, uint32_t wait_polls) {
    using Cf = ExtractCfg<H>;
    using W = typename Cf::W;
    constexpr int T = W::T, E = W::E, P = Cf::P, K = win_edge<H>();
    extern __shared__ __align__(16) float2 sm[];
    const int tr = threadIdx.x / T, j = threadIdx.x % T;
    const int a = blockIdx.y;
    const int ya = 2 * (blockIdx.x * P + tr), yb = ya + 1;
    float2* s = sm + tr * W::STRIDE;
    const float ha = 0.5f * __ldg(&win[ya]).x, hb = 0.5f * __ldg(&win[yb]).x;  // (-1)^y w(y) / 2
    const float2 flat = (j & 1) ? make_float2(-1.0f, 8388608.0f) : make_float2(1.0f, -8388608.0f);
    const size_t bpp = bits == 16 ? 2 : 1;
    float2 x[E];
    // windowed pixels of rows ya (real part) and yb (imaginary part)
    auto put = [&](int n1, uint32_t pa, uint32_t pb) {
        const float2 wc = (n1 < K || n1 >= E - K) ? __ldg(&win[j + n1 * T]) : flat;
        x[n1] = make_float2(fmaf(__uint_as_float(0x4B000000u | pa), wc.x, wc.y),
                            fmaf(__uint_as_float(0x4B000000u | pb), wc.x, wc.y));
    };
    auto load = [&](const char* row) {
        if (bits == 16) {
            const uint16_t* ra = reinterpret_cast<const uint16_t*>(row);
#pragma unroll
            for (int n1 = 0; n1 < E; ++n1) put(n1, ra[j + n1 * T], ra[H + j + n1 * T]);
        } else {
            const uint8_t* ra = reinterpret_cast<const uint8_t*>(row);
#pragma unroll
            for (int n1 = 0; n1 < E; ++n1) put(n1, ra[j + n1 * T], ra[H + j + n1 * T]);
        }
        if (ref_inv) {  // pixel / reference amplitude (it scales each product)
            const float* qa = ref_inv + (size_t)ya * H;
#pragma unroll
            for (int n1 = 0; n1 < E; ++n1) {
                const int xx = j + n1 * T;
                x[n1] = make_float2(x[n1].x * __ldg(&qa[xx]), x[n1].y * __ldg(&qa[H + xx]));
            }
        }
    };
    if constexpr (BULK) {
        __shared__ uint64_t bar[Cf::NT / 32];
        const int w = threadIdx.x >> 5;
        static_assert(2 * W::G * H * 2 + 8 <= W::STRIDE * 8, "staged rows fit the first array");
        // the warp's rows land at the first 16-byte boundary of its first
        // transform's array (8 (H + E + 1) bytes, so 2G H bpp + 8 fit), which
        // the transforms overwrite only after all lanes have read their pixels
        // (the first exchange follows a __syncwarp); the pointer is formed by
        // arithmetic on sm (no integer round trip), so the reads stay
        // shared-memory loads
        float2* const first = sm + (w * W::G) * W::STRIDE;
        char* stage = reinterpret_cast<char*>(first) + ((16u - (smem_addr(first) & 15u)) & 15u);
        if ((threadIdx.x & 31) == 0) {
            const uint32_t bytes = (uint32_t)(2 * W::G * H * bpp);
            const size_t y0w = 2 * ((size_t)blockIdx.x * P + w * W::G);
            mbar_init(&bar[w]);
            mbar_expect_tx(&bar[w], bytes);
            bulk_g2s(stage, static_cast<const char*>(holos) + ((size_t)a * H * H + y0w * H) * bpp, bytes, &bar[w]);
        }
        __syncwarp();
        if (!mbar_wait(&bar[w], 0, wait_polls)) {
            if ((threadIdx.x & 31) == 0) atomicOr(err, 2);
            mbar_wait(&bar[w], 0);
        }
        load(stage + (size_t)(tr - w * W::G) * 2 * H * bpp);
    } else {
        load(static_cast<const char*>(holos) + ((size_t)a * H * H + (size_t)ya * H) * bpp);
    }
    fft_warp_regs<H, -1>(x, s, j, tw);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < E / T; ++q) {
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) s[warp_out_pos<H>(j, q, k2)] = x[q * T + k2];
    }
    __syncwarp();
    // separate the two real rows on the kx band: Xa = (Z(k) + conj Z(-k))/2, Xb = (Z(k) - conj Z(-k))/(2i),
    // times the rows' window factors
    float2* dst = inter + ((size_t)a * H + ya) * F;
#pragma unroll 4
    for (int c = j; c < F; c += T) {
        const int k = x0 + c, km = (H - k) & (H - 1);
        const float2 z = s[W::pad(k)], zm = s[W::pad(km)];
        dst[c] = make_float2(ha * (z.x + zm.x), ha * (z.y - zm.y));
        dst[F + c] = make_float2(hb * (z.y + zm.y), -hb * (z.x - zm.x));
    }
}

template <int H>
__global__ void __launch_bounds__(ExtractCfg<H>::Cols::NT, ExtractCfg<H>::COLS_CTAS)
k_extract_cols(const float2* __restrict__ inter, const float2* __restrict__ tw, float2* __restrict__ spectra,
               float2* __restrict__ also, int F, int x0, int y0, float4* __restrict__ argpart) {
    using C = typename ExtractCfg<H>::Cols;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ __align__(16) float2 sm[];
    const int t = C::column(), j = C::adjacent_j();
    const int a = blockIdx.y, c = blockIdx.x * C::B + t;
    const bool valid = c < F;  // the crop width need not be a multiple of the columns
    const float2* src = inter + (size_t)a * H * F + c;
    float2 x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) x[n1] = valid ? src[(size_t)(j + n1 * T) * F] : make_float2(0.f, 0.f);
    fft_cta_regs<H, -1>(x, sm + t * W::STRIDE, j, tw);
    // (-1)^(kx+ky) / H^2: ky has j's parity
    const float inv = 1.0f / ((float)H * (float)H), sg = ((x0 + c + j) & 1) ? -inv : inv;
    float2* dst = spectra + (size_t)a * F * F + c;
    float best = -1.0f, second = -1.0f;
    int bi = 0x7fffffff;
    dst += (ptrdiff_t)(j - y0) * F;
    constexpr int GR = E >= 32 ? 4 : 2;  // output blocks of E rows tested for the crop together
#pragma unroll
    for (int g = 0; g < T / GR; ++g) {
        if (E * GR * (g + 1) <= y0 || E * GR * g >= y0 + F) continue;
#pragma unroll
        for (int k = 0; k < GR; ++k) {
#pragma unroll
            for (int q = 0; q < E / T; ++q) {
                const int k2 = g * GR + k, r = j + q * T + E * k2 - y0;  // crop row
                if (valid && (unsigned)r < (unsigned)F) {
                    const float2 z = c_scale(x[q * T + k2], sg);
                    dst[(ptrdiff_t)(q * T + E * k2) * F] = z;
                    if (also) also[(size_t)a * F * F + (size_t)r * F + c] = z;
                    if (argpart) argmax_take(best, bi, second, z, r * F + c);
                }
            }
        }
    }
    if (argpart) {  // this warp's partial winner of the specular search
        argmax_warp(best, bi, second);
        if ((threadIdx.x & 31) == 0)
            argpart[((size_t)a * gridDim.x + blockIdx.x) * (C::NT / 32) + (threadIdx.x >> 5)] =
                argmax_record(best, bi, second);
    }
}

}  // namespace extract
}  // namespace tdm
