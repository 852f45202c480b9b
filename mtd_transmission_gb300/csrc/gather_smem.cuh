// Shared memory of the cap gather (k_gather, k_recon.cu): its layout, the form a
// launch takes, and the angle limit of a context.  Host arithmetic besides the
// offsets, so that the rule can be checked without a GPU.
#pragma once

#include <cstddef>
#include <cstdint>

#include "fft_core.cuh"

namespace tdm {

constexpr size_t kMaxSmemPerCta = 227 * 1024;  // a launch's dynamic and the kernel's static bytes together

// A listed angle: its specular x and its index.  Both fit 16 bits: an angle is
// listed only when its window meets the CTA's columns, which bounds x by the
// volume's side, and a stack has at most 65535 angles.
struct Listed {
    int16_t x;
    uint16_t angle;
};

template <int W>
struct GatherSmem {
    // per warp: sums, counts (uint16) and cells with a hit (uint16), at a pitch of
    // 16 bytes mod 128: with the normalised cell of an odd plane in the upper half of its sums' slot, the
    // CTA-wide store's reads fall in distinct banks.  Per CTA: two tiles of 32
    // angles' cells (odd row pitches, so that a column is read without
    // conflicts) and the list of angles.
    static constexpr int VP = W + 1, ZP = W + 2;  // row pitches of a tile's values and planes
    static constexpr int TILE = 32 * VP * 8 + 32 * ZP * 2;
    static constexpr size_t STATIC = 2 * 32 * sizeof(unsigned);  // the listing's ballots
    __host__ __device__ static int cnt_at(int band) { return band * 16; }
    __host__ __device__ static int touched_at(int band) { return cnt_at(band) + ((band * 2 + 15) & ~15); }
    __host__ __device__ static int pitch(int band) {
        return ((touched_at(band) + ((band * 2 + 15) & ~15) - 16 + 127) & ~127) + 16;
    }
    __host__ __device__ static size_t bytes(int band, int n) {
        return (size_t)W * pitch(band) + 2 * TILE + (size_t)n * sizeof(Listed);
    }
    static bool fits(int band, int n) { return bytes(band, n) + STATIC <= kMaxSmemPerCta; }
};

// Columns (warps) of a CTA for n angles of a cap band of `band` planes; 0: no
// form fits.  16 where counts of a volume well beyond L2 are stored (k_gather's
// comment has both sides), if the CTA has room for them.
inline int gather_columns(int D, int band, int n, bool counts) {
    if (counts && D >= 512 && GatherSmem<16>::fits(band, n)) return 16;
    return GatherSmem<8>::fits(band, n) ? 8 : 0;
}

// The angle limit of a context: an angle count is accepted while a list of
// 8-byte entries fits a CTA's shared memory beside the FP64 sums and counts of
// four warps' columns (two columns a warp up to D = 512, whose FFT takes half a
// warp), or their FFT exchange buffers, the plane owners, a staging row and
// the mask bits.  k_gather, with 4-byte entries, needs less for every band
// (at most sqrt(2) F + 2 planes, F <= 512) and count that this accepts.
inline size_t gather_limit_bytes(int D, int band, int n) {
    const int T = D / warp_fft_e(D), G = 32 / T;
    const size_t sums = (size_t)G * band * (sizeof(double2) + sizeof(uint16_t)), xch = (size_t)G * T * (T + 1) * sizeof(float2);
    const size_t region = ((sums > xch ? sums : xch) + 15) & ~size_t(15);
    return 4 * (region + 32 * sizeof(float2) + ((band + 15) & ~15)) + (((size_t)band * 4 + 7) & ~size_t(7)) +
           (size_t)n * sizeof(int2);
}

}  // namespace tdm
