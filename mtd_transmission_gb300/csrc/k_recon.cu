// Reconstruction (Reconstruction/main.cpp:203-352).
//
// Per field (main.cpp:207-217): x Tukey(0.1), shift by (N, N), forward FFT x dx^2,
// shift by posSpec.  With k the FFT bin, the value that retroPropag_Born reads
// at cap pixel fd = ((k + posSpec) mod F) - N is
//     (-1)^(kx+ky) dx^2 FFT2(field * tukey)[k],
// so the per-field kernels work on natural FFT bins and store, per bin, the
// cap contribution -2i k0 sdz value (cteUb2Pot*cteNorm*sdz, fonctions.cpp:902,927),
// 0 outside the cap cells (an 8-byte cap value), and the cell's volume plane z
// (-1 outside the NA disc) as a 2-byte integer: the gather reads the planes of
// the bins that fall in its column and the values of the cells that hit it.
//
// Mapping (retroPropag_Born, src/fonctions.cpp:875-935) as a gather: voxel
// column (X, Y) reads bin kx = (X - D/2) mod F for every angle whose cap window
// covers it; each angle hits a column at most once, so the column's sums are
// formed without atomics, in a fixed order; hit counts are exact (k_gather).
//
// Volume: fftshift3D, backward 3D FFT x Delta_f^3, fftshift3D, x -1/(2 n0 kv^2)
// (main.cpp:282-352).  For even D the two shifts are sign modulations:
//     out[m] = (-1)^(mx+my+mz+3D/2) IFFT3((-1)^(kx+ky+kz) V)[m].
// Caps reach only `band` of the D planes, and only the columns within F of the
// centre, so the spectrum is kept as its band planes ([e][y][x], e = z - zmin)
// and the transform along z comes last: the x and y passes run on band planes
// only, and the z pass widens them to the D planes as it writes the index and
// absorption volumes.  At 600 angles, 256^2 fields, 512^3 (band 220) the
// stage moves 3.8 GB where transforming z first, over all columns, moved
// 5.4 GB.
#include "tdm_internal.cuh"
#include "fft_warp.cuh"
#include "form.cuh"
#include "fp_bits.cuh"
#include "cap_geometry.cuh"
#include "gather_smem.cuh"
#include "quotient.cuh"

namespace tdm {
namespace {

template <class K>
cudaError_t allow_smem(K kernel, size_t bytes) {
    return max_dynamic_smem(reinterpret_cast<const void*>(kernel), bytes);
}

template <int F>
struct CapCfg {
    using W = WarpFFT<F>;
    static constexpr int B = 8 * W::G;    // transforms per CTA
    static constexpr int NT = B * W::T;   // 256 threads
    static constexpr size_t SMEM = (size_t)B * W::STRIDE * sizeof(float2);
};

// copy (may be null) receives the fields.
template <int F>
__global__ void __launch_bounds__(CapCfg<F>::NT)
k_cap_rows(const float2* __restrict__ fields, const float* __restrict__ tuk, int2 flat, const float2* __restrict__ tw,
           float2* __restrict__ r1, float2* __restrict__ copy) {
    using C = CapCfg<F>;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ float2 sm[];
    const int tr = threadIdx.x / T, j = threadIdx.x % T;
    const int a = blockIdx.y, y = blockIdx.x * C::B + tr;
    const float wy = tuk[y];
    const float2* src = fields + ((size_t)a * F + y) * F;
    Fusable x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) {
        const int xx = j + n1 * T;
        x[n1] = src[xx];
    }
    if (copy) {
#pragma unroll
        for (int n1 = 0; n1 < E; ++n1) copy[((size_t)a * F + y) * F + j + n1 * T] = x[n1];
    }
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) {
        const int xx = j + n1 * T;
        x[n1] = c_scale(x[n1], ((xx >= flat.x && xx <= flat.y) ? 1.0f : __ldg(&tuk[xx])) * wy);
    }
    fft_warp_regs<F, -1>(x, sm + tr * W::STRIDE, j, tw);
    float2* dst = r1 + ((size_t)a * F + y) * F;
#pragma unroll
    for (int q = 0; q < E / T; ++q) {
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) dst[j + q * T + E * k2] = x[q * T + k2];
    }
}

// k_cap_rows with the field formed on the fly from the chunk's unwrapped
// phase, amplitude and fits (the field stage's k_form, same arithmetic); the
// field is also stored, as k_form would.
template <int F>
__global__ void __launch_bounds__(CapCfg<F>::NT)
k_cap_rows_form(const float* __restrict__ unwrapped, const float* __restrict__ amp, const double* __restrict__ beta,
                int born, const float* __restrict__ tuk, int2 flat, const float2* __restrict__ tw,
                float2* __restrict__ fields,
                float2* __restrict__ r1) {
    using C = CapCfg<F>;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ float2 sm[];
    __shared__ float bf[2 * kNC];
    if (threadIdx.x < 2 * kNC) bf[threadIdx.x] = (float)beta[(size_t)blockIdx.y * 2 * kNC + threadIdx.x];
    __syncthreads();
    const int tr = threadIdx.x / T, j = threadIdx.x % T;
    const int a = blockIdx.y, y = blockIdx.x * C::B + tr;
    const float wy = tuk[y];
    const size_t row = ((size_t)a * F + y) * F;
    const FormRow fr = form_row(bf, y, F);
    Fusable x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) {
        const int xx = j + n1 * T;
        const float2 f = form_value(fr, xx, F, unwrapped[row + xx], amp[row + xx], born);
        fields[row + xx] = f;
        x[n1] = c_scale(Fusable(f), ((xx >= flat.x && xx <= flat.y) ? 1.0f : __ldg(&tuk[xx])) * wy);
    }
    fft_warp_regs<F, -1>(x, sm + tr * W::STRIDE, j, tw);
    float2* dst = r1 + row;
#pragma unroll
    for (int q = 0; q < E / T; ++q) {
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) dst[j + q * T + E * k2] = x[q * T + k2];
    }
}

// Column passes (ColFFT) with at least 512 threads an SM: 128 registers each.
template <int D>
struct ColPass : ColFFT<D> {
    using ColFFT<D>::NT;
    static constexpr int CTAS = NT <= 128 ? 4 : NT <= 256 ? 2 : 1;
};

// Columns of the per-field spectrum (ColFFT) and their cap records.
template <int F>
__global__ void __launch_bounds__(ColFFT<F>::NT, 512 / ColFFT<F>::NT)
k_cap_cols(const float2* __restrict__ r1, const int2* __restrict__ posspec, const double* __restrict__ s_tab,
           const float2* __restrict__ s_pair, Params p, const float2* __restrict__ tw, float2* __restrict__ rec,
           int16_t* __restrict__ recz, int* __restrict__ err) {
    using C = ColFFT<F>;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ float2 sm[];
    const int t = C::column(), j = C::adjacent_j();
    const int a = blockIdx.y, kx = blockIdx.x * C::B + t;
    const int2 ps = posspec[a];
    const CapFz fz = cap_fzm0(p, ps, s_tab, s_pair);
    const float ir = (float)p.inv_rayon;
    const size_t o = (size_t)a * F * F + kx;
    Fusable x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) x[n1] = r1[o + (size_t)(j + n1 * T) * F];
    fft_cta_regs<F, -1>(x, sm + t * W::STRIDE, j, tw);
    auto put = [&](int ky, float2 v) {
        float sf = 0.f;
        const int z = cap_plane(p, ps, fz, kx, ky, s_tab, s_pair, &sf, err);
        float2 val = make_float2(0.f, 0.f);
        if (z >= 0) {
            const float Bc = cap_weight(p, sf, ir, kx, ky);
            val = make_float2(-Bc * v.y, Bc * v.x);
        }
        rec[o + (size_t)ky * F] = val;
        recz[o + (size_t)ky * F] = (int16_t)z;
    };
    if constexpr (E <= 16) {
#pragma unroll
        for (int q = 0; q < E / T; ++q) {
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) put(j + q * T + E * k2, x[q * T + k2]);
        }
    } else {
        // 32 unrolled bins take 246 registers (194 us for 64 angles of 512^2, against 148 as below): the
        // thread's values wait in its own places of the exchange array instead
        float2* s = sm + t * W::STRIDE;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < E / T; ++q) {
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) s[warp_out_pos<F>(j, q, k2)] = x[q * T + k2];
        }
#pragma unroll 2
        for (int i = 0; i < E; ++i) {
            const int q = i / T, k2 = i % T;
            put(j + q * T + E * k2, s[warp_out_pos<F>(j, q, k2)]);
        }
    }
}

// ---------------------------------------------------------------- cap accumulation
// One warp per voxel column (X, Y).  An angle's cap window is the F x F bins
// around its specular position, so a column is covered by a fraction of the
// angles: a CTA first lists, in ascending order, the angles whose window covers
// its row Y and any of its columns, and takes them 32 at a time: its threads
// load the 32 angles' cells of its columns (the plane, a 2-byte record, and the
// cap value), neighbouring threads neighbouring columns, into a shared-memory
// tile, the next 32 angles' cells on their way meanwhile, and a warp's lanes
// then read its column's cells of the 32 angles.  (With the lanes loading their
// angles' records themselves, every lane another line, the L1's data pipe was 85 %
// busy and bounded the gather: 600 angles of 256^2 to 512^3 518 us.)  Groups
// without a hit are skipped.  An angle hits a column at most once, at one plane.
//
// A column's running sums live in shared memory as pairs of floats: each hit is
// added to the first by an error-free sum (Knuth's two-sum, on packed pairs of
// real and imaginary part) whose error goes to the second, about 2^-48 of the
// largest partial sum in all, where FP64 sums of FP32 group sums (the hits of 32
// angles at one plane added in FP32 first) had that of an FP32 sum; FP64 adds run
// at 1/64 of the FP32 rate here.  (Error of 600 random hits' sum, rounded to FP32:
// 2.5e-8 relative, 3.2e-5 before; of positive hits 2.4e-8 and 2.5e-8.)  Hits of a group at the same plane are added
// one after the other in ascending angle order, so the sums are deterministic;
// the hit counts are exact.

// Lists, in ascending order, the angles whose window covers row Y (by = Y -
// D/2) and one of the columns bx0 .. bx0 + nx - 1 of the CTA.  Returns the
// count; all NW warps of the CTA call it together, and it ends with a barrier.
// 1024 angles a round: each warp tests its share in 32-angle pieces, and after
// one barrier every warp scans the 32 pieces' ballots for the places of its own.
template <int NW>
__device__ __forceinline__ int list_angles(const int2* __restrict__ posspec, int M, int F, int by, int bx0, int nx,
                                           Listed* list, unsigned (*s_bal)[32]) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int K = 32 / NW;  // pieces per warp and round
    int base = 0;
    for (int a0 = 0, r = 0; a0 < M; a0 += 1024, r ^= 1) {
        int qx[K];
        unsigned bal[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int a = a0 + (k * NW + w) * 32 + lane;
            bool keep = false;
            qx[k] = 0;
            if (a < M) {
                const int2 q = posspec[a];
                keep = (unsigned)(by + q.y) < (unsigned)F && bx0 + nx - 1 + q.x >= 0 && bx0 + q.x < F;
                qx[k] = q.x;
            }
            bal[k] = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) s_bal[r][k * NW + w] = bal[k];
        }
        __syncthreads();  // the other round's ballots are read before the barrier after next
        const int own = __popc(s_bal[r][lane]);
        int incl = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int off = base + __shfl_sync(0xffffffffu, incl - own, k * NW + w);
            if ((bal[k] >> lane) & 1u)
                list[off + __popc(bal[k] & ((1u << lane) - 1u))] =
                    Listed{(int16_t)qx[k], (uint16_t)(a0 + (k * NW + w) * 32 + lane)};
        }
        base += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncthreads();
    return base;
}

// A column's sums: acc (x, y: the sum; z, w: its error) is valid where cnt is not
// 0; touched lists the `hit` cells with a hit.
struct ColumnSums {
    float4* acc;
    uint16_t *cnt, *touched;
    int hit;
};

// One warp adds 32 angles' cells of its column to the column's sums: this
// lane's cell has plane z (or -1) and value v; lane l's value is vs[l * pitch].
// The first lane at a plane adds the values of all lanes there.
__device__ __forceinline__ void gather_add(ColumnSums& c, int z, float2 v, const float2* vs, int pitch, int zmin,
                                           int lane) {
    const int e = z >= 0 ? z - zmin : -1;
    if (!__any_sync(0xffffffffu, e >= 0)) return;
    const unsigned same = __match_any_sync(0xffffffffu, e), below = (1u << lane) - 1u;
    const bool leads = e >= 0 && !(same & below);
    const unsigned n = leads ? c.cnt[e] : 1;
    const unsigned fresh = __ballot_sync(0xffffffffu, n == 0);
    if (leads) {
        float2 hi = v, lo = make_float2(0.f, 0.f);
        auto add = [&](float2 u) {
            const float2 s = c_add(hi, u), b = c_sub(s, hi);
            lo = c_add(lo, c_add(c_sub(hi, c_sub(s, b)), c_sub(u, b)));
            hi = s;
        };
        if (n) {
            const float4 t = c.acc[e];
            hi = make_float2(t.x, t.y), lo = make_float2(t.z, t.w);
            add(v);
        } else {
            c.touched[c.hit + __popc(fresh & below)] = (uint16_t)e;
        }
        for (unsigned g = same & ~below & ~(1u << lane); g; g &= g - 1) add(vs[(__ffs(g) - 1) * pitch]);
        c.acc[e] = make_float4(hi.x, hi.y, lo.x, lo.y);
        c.cnt[e] = (uint16_t)(n + __popc(same));
    }
    c.hit += __popc(fresh);
    __syncwarp();
}

// k_gather: a CTA of W warps takes W consecutive columns at one Y.  Each warp
// normalises its column's cells in place (not normalised for the adjoint
// scatter; (-1)^(X+Y+Z) stands for the first fftshift3D), and the CTA stores the
// columns together as rows of consecutive x of the [e][y][x] spectrum, with the
// OTF mask (Re != 0 after normalisation, main.cpp:262-267) and the counts, which
// one column at a time would scatter plane by plane.  The grid covers the columns
// that caps can reach; cells outside them and outside the band are cleared by
// the host.  8 columns a CTA, for more warps an SM; with the counts of a volume
// well beyond L2 16 columns, whose rows of counts are whole 64-byte pieces (300
// angles of 256^2 to 512^3 418 -> 381 us, 64 of 512^2 to 1024^3 3.5 -> 2.3 ms; at
// 256^3 8 columns take 76 us, 16 90).
//
// Bound by issue and latency (64 angles, 8 columns a CTA: issue 77 % active at 59 % of
// the warps; six CTAs an SM leave 40 registers, and 20 bytes are spilled).  600 angles of 256^2 to 512^3: 434 us (with FP64
// sums of FP32 group sums, and each lane loading its angle's records, 538); 400
// of 128^2 to 256^3 76 us (100).
template <int W>
__global__ void __launch_bounds__(W * 32, W == 8 ? 6 : 2)
k_gather(const float2* __restrict__ rec, const int16_t* __restrict__ recz, const int2* __restrict__ posspec, int M,
         Params p, float2* __restrict__ vol, uint32_t* __restrict__ cnt_out, uint8_t* __restrict__ otf,
         int normalize) {
    using S = GatherSmem<W>;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ unsigned s_bal[2][32];
    static_assert(sizeof(s_bal) == S::STATIC, "the form's choice counts it");
    const int band = p.band, F = p.F, D = p.D, h = D / 2, zmin = p.zmin;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pitch = S::pitch(band), cnt_at = S::cnt_at(band);
    unsigned char* mine = smraw + w * pitch;
    ColumnSums col{reinterpret_cast<float4*>(mine), reinterpret_cast<uint16_t*>(mine + cnt_at),
                   reinterpret_cast<uint16_t*>(mine + S::touched_at(band)), 0};
    unsigned char* tile = smraw + W * pitch;
    Listed* list = reinterpret_cast<Listed*>(tile + 2 * S::TILE);
    auto cell = [](unsigned char* c, int e) { return reinterpret_cast<float2*>(c + e * 16 + (e & 1) * 8); };
    const size_t FF = (size_t)F * F, plane = (size_t)D * D;
    const int X0 = p.xa + blockIdx.x * W, Y = p.ya + blockIdx.y, by = Y - h;
    for (int e = lane; e < (band + 1) / 2; e += 32) reinterpret_cast<uint32_t*>(col.cnt)[e] = 0;
    const int listed = list_angles<W>(posspec, M, F, by, X0 - h, W, list, s_bal);
    // this thread's cell of a group of 32 listed angles: column c, angle i of the group
    const int c = threadIdx.x % W, i = threadIdx.x / W, bx = X0 + c - h;
    const size_t koff = (size_t)(((by % F) + F) % F) * F + ((bx % F) + F) % F;
    float2 v = make_float2(0.f, 0.f);
    int z = -1;
    auto fetch = [&](int g0) {
        z = -1;
        if (g0 + i < listed) {
            const Listed q = list[g0 + i];
            if ((unsigned)(bx + q.x) < (unsigned)F) {  // the angle's window covers the column
                const size_t o = (size_t)q.angle * FF + koff;
                z = __ldg(&recz[o]);
                v = __ldg(&rec[o]);
            }
        }
    };
    fetch(0);
    for (int g0 = 0, k = 0; g0 < listed; g0 += 32, k ^= 1) {
        float2* tv = reinterpret_cast<float2*>(tile + k * S::TILE);
        int16_t* tz = reinterpret_cast<int16_t*>(tv + 32 * S::VP);
        tv[i * S::VP + c] = v;
        tz[i * S::ZP + c] = (int16_t)z;
        fetch(g0 + 32);
        __syncthreads();  // the other tile is read before the barrier after this one
        gather_add(col, tz[lane * S::ZP + w], tv[lane * S::VP + w], tv + w, S::VP, zmin, lane);
    }
    for (int t = lane; t < col.hit; t += 32) {
        const int e = col.touched[t];
        const float4 sum = col.acc[e];
        float2 u = make_float2(sum.x + sum.z, sum.y + sum.w);
        // an infinite sum has no error term
        if (!(u.x == u.x)) u.x = sum.x;
        if (!(u.y == u.y)) u.y = sum.y;
        if (normalize) {
            const float n = (float)col.cnt[e], r = __frcp_rn(n);
            u = make_float2(over(u.x, n, r), over(u.y, n, r));
        }
        *cell(mine, e) = ((X0 + w + Y + zmin + e) & 1) ? make_float2(-u.x, -u.y) : u;
    }
    __syncthreads();
    unsigned char* from = smraw + c * pitch;
    size_t o = (size_t)Y * D + X0 + c + i * plane;
    for (int e = i; e < band; e += 32, o += 32 * plane) {
        const unsigned n = reinterpret_cast<uint16_t*>(from + cnt_at)[e];
        const float2 u = n ? *cell(from, e) : make_float2(0.f, 0.f);
        vol[o] = u;
        if (cnt_out) cnt_out[zmin * plane + o] = n;
        if (otf) otf[zmin * plane + o] = u.x != 0.0f;
    }
}

// ---------------------------------------------------------------- 3D FFT passes
// Column passes (y, z): ColFFT, 16 consecutive x a CTA.  Bound by HBM: 512^3
// with a band of 220, x 137 us and y 144 us (6.7 and 6.4 TB/s), z 293 us
// (5.2 TB/s, most of it stores); over all planes and staged through shared memory
// y and x took 405 and 432 us.  8 columns leave 32-byte pieces in the z pass's
// stores (713 us), 32 one CTA an SM (y 182, z 352 us).

// Row pass (x): a warp per G rows, registers to registers.
template <int D>
struct RowPass {
    using W = WarpFFT<D>;
    static constexpr int B = 8 * W::G;
    static constexpr int NT = 256;
    static constexpr size_t SMEM = (size_t)B * W::STRIDE * sizeof(float2);
};

// FFT along x of the band planes' rows in [ya, yb), in place.  Inverse (DIR
// +1): columns outside [xa, xb) hold nothing and are taken as zero.  Forward:
// the last pass of the forward operator, x (-1)^(X+Y+Z), only [xa, xb) written.
template <int D, int DIR>
__global__ void __launch_bounds__(RowPass<D>::NT, 2)
k_xpass(float2* __restrict__ vol, const float2* __restrict__ tw, Params p) {
    using C = RowPass<D>;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ float2 sm[];
    const int tr = threadIdx.x / T, j = threadIdx.x % T;
    const int ny = p.yb - p.ya;
    int r = blockIdx.x * C::B + tr;  // band row: plane e, row Y
    const bool ok = r < p.band * ny;
    if (!ok) r = 0;
    const int e = r / ny, Y = p.ya + r % ny;
    float2* row = vol + ((size_t)e * D + Y) * D;
    float2 x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) {
        const int X = j + n1 * T;
        x[n1] = DIR < 0 || (X >= p.xa && X < p.xb) ? row[X] : make_float2(0.f, 0.f);
    }
    fft_warp_regs<D, DIR>(x, sm + tr * W::STRIDE, j, tw);
    if (!ok) return;
    const float sg = DIR < 0 && ((j + Y + p.zmin + e) & 1) ? -1.0f : 1.0f;  // X has j's parity
#pragma unroll
    for (int q = 0; q < E / T; ++q) {
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) {
            const int X = j + q * T + E * k2;
            const float2 v = x[q * T + k2];
            if (DIR > 0) row[X] = v;
            else if (X >= p.xa && X < p.xb) row[X] = make_float2(v.x * sg, v.y * sg);
        }
    }
}

// FFT along y of the band planes, in place; inverse: rows outside [ya, yb)
// are taken as zero; forward: only rows in [ya, yb) are written.
template <int D, int DIR>
__global__ void __launch_bounds__(ColPass<D>::NT, ColPass<D>::CTAS)
k_ypass(float2* __restrict__ vol, const float2* __restrict__ tw, Params p) {
    using C = ColPass<D>;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ float2 sm[];
    const int t = C::column(), j = C::adjacent_j();
    float2* col = vol + (size_t)blockIdx.y * D * D + blockIdx.x * C::B + t;
    float2 x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) {
        const int Y = j + n1 * T;
        x[n1] = DIR < 0 || (Y >= p.ya && Y < p.yb) ? col[(size_t)Y * D] : make_float2(0.f, 0.f);
    }
    fft_cta_regs<D, DIR>(x, sm + t * W::STRIDE, j, tw);
#pragma unroll
    for (int q = 0; q < E / T; ++q) {
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) {
            const int Y = j + q * T + E * k2;
            if (DIR > 0 || (Y >= p.ya && Y < p.yb)) col[(size_t)Y * D] = x[q * T + k2];
        }
    }
}

// The z pass's stores: a volume well beyond L2, which its reader cannot find there
// again, is stored to be evicted first and leaves the cache to the planes that are
// read (512^3 325 -> 293 us; 1024^3 3.29 ms before, 3.22 to 3.34 after).  It gave
// nothing to the x and y passes (x 138 -> 134, y 141 -> 143 us), whose 461 MB the
// next pass reads.
template <int D>
__device__ __forceinline__ void put(float* q, float v) {
    if constexpr (D >= 512) __stcs(q, v);
    else *q = v;
}

// Inverse FFT along z of the band (zero elsewhere), scaled and
// sign-modulated, written as the index (real) and absorption (imaginary)
// volumes (either may be null), x fastest.
template <int D>
__global__ void __launch_bounds__(ColPass<D>::NT, ColPass<D>::CTAS)
k_zpass(const float2* __restrict__ vol, const float2* __restrict__ tw, Params p, float scale, float* __restrict__ re,
        float* __restrict__ im) {
    using C = ColPass<D>;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ float2 sm[];
    const int t = C::column(), j = C::adjacent_j();
    const int X = blockIdx.x * C::B + t, Y = blockIdx.y;
    const float2* col = vol + (size_t)Y * D + X;
    float2 x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) {
        const int e = j + n1 * T - p.zmin;
        x[n1] = (unsigned)e < (unsigned)p.band ? col[(size_t)e * D * D] : make_float2(0.f, 0.f);
    }
    fft_cta_regs<D, +1>(x, sm + t * W::STRIDE, j, tw);
    const float sg = ((X + Y + j + 3 * (D / 2)) & 1) ? -scale : scale;  // z has j's parity
    const size_t o = (size_t)Y * D + X;
#pragma unroll
    for (int q = 0; q < E / T; ++q) {
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) {
            const size_t z = j + q * T + E * k2;
            if (re) put<D>(&re[z * D * D + o], x[q * T + k2].x * sg);
            if (im) put<D>(&im[z * D * D + o], x[q * T + k2].y * sg);
        }
    }
}

// ---------------------------------------------------------------- forward operator and adjoint
// With the unknown volume x = index + i absorption ([z][y][x], x fastest) and
// s = out_scale, the volume stage above is x = T(V) = s M_out IFFT3(M_in V)
// (unnormalised IFFT, M the fftshift sign patterns).  The forward operator
// is A = S G with G = T^-1 = M_in FFT3(M_out x) / (s D^3) and S the sampling
// of each angle's cap cells (the cells the gather fills, same geometry); its
// adjoint is A^H = G^H S^H, G^H = M_out IFFT3(M_in .) / (s D^3) and S^H the
// unnormalised scatter, i.e. k_gather without the division by the hit
// count, followed by the x, y and z passes with scale 1 / (s D^3).

// Forward z pass: FFT along z of the index/absorption volumes (x M_out x
// scale), only the cap band written (the sampling reads nothing else).
template <int D>
__global__ void __launch_bounds__(ColPass<D>::NT, ColPass<D>::CTAS)
k_fzpass(const float* __restrict__ re, const float* __restrict__ im, const float2* __restrict__ tw, Params p,
         float scale, float2* __restrict__ vol) {
    using C = ColPass<D>;
    using W = typename C::W;
    constexpr int T = W::T, E = W::E;
    extern __shared__ float2 sm[];
    const int t = C::column(), j = C::adjacent_j();
    const int X = blockIdx.x * C::B + t, Y = blockIdx.y;
    const size_t o = (size_t)Y * D + X;
    const float sg = ((X + Y + j + 3 * (D / 2)) & 1) ? -scale : scale;  // z has j's parity
    float2 x[E];
#pragma unroll
    for (int n1 = 0; n1 < E; ++n1) {
        const size_t z = j + n1 * T;
        x[n1] = make_float2(re[z * D * D + o] * sg, im ? im[z * D * D + o] * sg : 0.0f);
    }
    fft_cta_regs<D, -1>(x, sm + t * W::STRIDE, j, tw);
#pragma unroll
    for (int q = 0; q < E / T; ++q) {
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) {
            const int e = j + q * T + E * k2 - p.zmin;
            if ((unsigned)e < (unsigned)p.band) vol[(size_t)e * D * D + o] = x[q * T + k2];
        }
    }
}

// Cap values of the spectrum: for each angle and FFT bin, the spectrum at its
// cap cell (0 outside the cap).  With data (cap values of measurements), the
// residual spectrum - data on the cap cells (0 elsewhere) and the misfit
// sum |residual|^2 added to *misfit.  (8 bytes are spilled around the call that
// computes a height outside the table, which caps inside the field do not make.)
__global__ void __launch_bounds__(256)
k_cap_sample(const float2* __restrict__ vol, const int2* __restrict__ posspec, Params p,
             const double* __restrict__ s_tab, const float2* __restrict__ s_pair, const float2* __restrict__ data,
             float2* __restrict__ caps, float2* __restrict__ res, int16_t* __restrict__ resz, double* __restrict__ misfit,
             int* __restrict__ err) {
    const int a = blockIdx.y, F = p.F, D = p.D;
    const int2 ps = posspec[a];
    __shared__ double red[8];
    const CapFz fz = cap_fzm0(p, ps, s_tab, s_pair);
    double m2 = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < F * F; i += gridDim.x * blockDim.x) {
        const int kx = i % F, ky = i / F;
        const size_t o = (size_t)a * F * F + i;
        float sf;
        const int z = cap_plane(p, ps, fz, kx, ky, s_tab, s_pair, &sf, err);
        float2 v = make_float2(0.f, 0.f);
        if (z >= 0) {
            const float2 d = data ? data[o] : make_float2(0.f, 0.f);
            const int X = cap_col(p, kx, ps.x), Y = cap_col(p, ky, ps.y);
            v = vol[((size_t)(z - p.zmin) * D + Y) * D + X];
            v = make_float2(v.x - d.x, v.y - d.y);
            const double vx = widen(v.x), vy = widen(v.y);  // the FP64 pipe squares and adds only
            m2 = fma(vy, vy, fma(vx, vx, m2));
        }
        if (caps) caps[o] = v;
        if (res) {
            res[o] = v;
            resz[o] = (int16_t)z;
        }
    }
    if (misfit) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) m2 += __shfl_down_sync(0xffffffffu, m2, off);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m2;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
            atomicAdd(misfit, t);
        }
    }
}

// Cap values of given values on the cap cells (0 elsewhere), for the scatter.
__global__ void __launch_bounds__(256)
k_cap_pack(const float2* __restrict__ caps, const int2* __restrict__ posspec, Params p,
           const double* __restrict__ s_tab, const float2* __restrict__ s_pair, float2* __restrict__ rec,
           int16_t* __restrict__ recz, int* __restrict__ err) {
    const int a = blockIdx.y, F = p.F;
    const int2 ps = posspec[a];
    const CapFz fz = cap_fzm0(p, ps, s_tab, s_pair);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < F * F; i += gridDim.x * blockDim.x) {
        const size_t o = (size_t)a * F * F + i;
        float sf;
        const int z = cap_plane(p, ps, fz, i % F, i / F, s_tab, s_pair, &sf, err);
        const float2 v = z >= 0 ? caps[o] : make_float2(0.f, 0.f);
        rec[o] = v;
        recz[o] = (int16_t)z;
    }
}

// One projected-gradient step of the regularised reconstruction, per voxel of
// the [z][y][x] volumes: x <- clamp(x - step g - tv dTV(x)), for the index
// (channel 0) and, when present, the absorption (channel 1).  TV is the
// isotropic total variation with forward differences (zero across the far
// faces) smoothed by eps: sum sqrt(|grad x|^2 + eps^2).  Its gradient at a
// voxel takes the cells anchored at the voxel and at its x, y and z
// predecessors.
//
// Bound by HBM (x and g read, x written: 12 bytes a voxel and channel; the
// neighbouring rows come from L1 and L2) and, with TV, by issue.  A thread
// takes four voxels of a row as 16-byte words and walks kTvPlanes planes in
// z, so that a plane's rows and cells serve the next one: three rows read
// and nine cells formed per four voxels, where one plane alone needs seven and
// sixteen.  The words' x neighbours come from the adjacent lanes, and from
// memory at the warp's ends only: D is a power of two of at least 128, so a
// warp's 128 voxels lie in one row, and a voxel's coordinates are shifts.
// 256^3, both channels: 106 us (3.8 TB/s of the 403 MB); the same words without
// the walk 130 us; one voxel per thread with its coordinates by 64-bit
// divisions 487 us.
struct TvChannel {
    const float *x, *g;
    float* out;
    float tv, lo, hi;
};

constexpr int kTvPlanes = 8;  // divides D

__global__ void __launch_bounds__(256)
k_tv_step(TvChannel c0, TvChannel c1, int log_d, float step, float eps2) {
    const TvChannel c = blockIdx.y ? c1 : c0;
    const int D = 1 << log_d, lane = threadIdx.x & 31;
    const size_t i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;  // voxel of the first plane, planes kTvPlanes apart
    const int X = (int)(i & (D - 1)), Y = (int)(i >> log_d) & (D - 1);
    const int Z0 = (int)(i >> (2 * log_d)) * kTvPlanes;
    const ptrdiff_t sy = D, sz = (ptrdiff_t)D * D;
    const size_t v0 = (size_t)Z0 * sz + (size_t)Y * sy + X;
    const bool y0 = Y > 0, y1 = Y + 1 < D, tv = c.tv != 0.0f;
    const float* xp = c.x + v0;
    // elements x - 1 .. x + 4 of a row in w[0 .. 5]; zeros where the row does not exist
    auto row = [&](float* w, bool ok, ptrdiff_t o) {
        const float4 q = ok ? *reinterpret_cast<const float4*>(xp + o) : make_float4(0.f, 0.f, 0.f, 0.f);
        w[1] = q.x, w[2] = q.y, w[3] = q.z, w[4] = q.w;
    };
    auto before = [&](float* w, bool ok, ptrdiff_t o) {
        w[0] = __shfl_up_sync(0xffffffffu, w[4], 1);
        if (lane == 0) w[0] = ok && X > 0 ? xp[o - 1] : 0.f;
    };
    auto after = [&](float* w, bool ok, ptrdiff_t o) {
        w[5] = __shfl_down_sync(0xffffffffu, w[1], 1);
        if (lane == 31) w[5] = ok && X + 4 < D ? xp[o + 4] : 0.f;
    };
    // the cell anchored at value ctr with successors nx, ny, nz (0 differences across the far faces)
    auto cell = [&](float ctr, float nx, float ny, float nz, bool okx, bool oky, bool okz, float& gx, float& gy,
                    float& gz) {
        gx = okx ? nx - ctr : 0.0f;
        gy = oky ? ny - ctr : 0.0f;
        gz = okz ? nz - ctr : 0.0f;
        return rsqrtf(gx * gx + gy * gy + gz * gz + eps2);
    };
    // rows (y, z), (y - 1, z) with their x neighbours; the z-predecessors' gz and 1 / norm
    float a[6], e[6], pz[4], pinv[4];
    row(a, true, 0);
    if (tv) {
        row(e, y0, -sy);
        before(a, true, 0), after(a, true, 0), after(e, y0, -sy);
        const bool z0 = Z0 > 0;
        float f[6], fu[6];
        row(f, z0, -sz);
        after(f, z0, -sz);
        row(fu, z0 && y1, sy - sz);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float gx, gy;
            pinv[k] = cell(f[k + 1], f[k + 2], fu[k + 1], a[k + 1], X + k + 1 < D, y1, true, gx, gy, pz[k]);
        }
    }
#pragma unroll 1
    for (int dz = 0; dz < kTvPlanes; ++dz) {
        const ptrdiff_t o = dz * sz;
        const int Z = Z0 + dz;
        const float4 gv = *reinterpret_cast<const float4*>(c.g + v0 + o);
        float r[4] = {a[1] - step * gv.x, a[2] - step * gv.y, a[3] - step * gv.z, a[4] - step * gv.w};
        const bool z1 = Z + 1 < D;
        float d[6];  // row (y, z + 1)
        row(d, z1 && (tv || dz + 1 < kTvPlanes), o + sz);
        if (tv) {
            float b[6], eu[6];  // rows (y + 1, z), (y - 1, z + 1)
            row(b, y1, o + sy);
            row(eu, y0 && z1, o + sz - sy);
            before(b, y1, o + sy), before(d, z1, o + sz);
            after(d, z1, o + sz), after(eu, y0 && z1, o + sz - sy);
            float gxp, gyp, gzp;  // the cell anchored at x - 1 + k
            float invp = cell(a[0], a[1], b[0], d[0], true, y1, z1, gxp, gyp, gzp);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool x1 = X + k + 1 < D;
                float gx, gy, gz, hx, hy, hz;
                const float inv = cell(a[k + 1], a[k + 2], b[k + 1], d[k + 1], x1, y1, z1, gx, gy, gz);
                float g = -(gx + gy + gz) * inv;
                if (X + k > 0) g += gxp * invp;
                const float invy = cell(e[k + 1], e[k + 2], a[k + 1], eu[k + 1], x1, true, z1, hx, hy, hz);
                if (y0) g += hy * invy;
                if (Z > 0) g += pz[k] * pinv[k];
                r[k] -= c.tv * g;
                gxp = gx, invp = inv, pz[k] = gz, pinv[k] = inv;
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) e[k] = eu[k];
        }
        *reinterpret_cast<float4*>(c.out + v0 + o) =
            make_float4(fminf(fmaxf(r[0], c.lo), c.hi), fminf(fmaxf(r[1], c.lo), c.hi),
                        fminf(fmaxf(r[2], c.lo), c.hi), fminf(fmaxf(r[3], c.lo), c.hi));
#pragma unroll
        for (int k = 0; k < 6; ++k) a[k] = d[k];
    }
}

template <int F>
int cap_impl(tdm_ctx* c, int a0, int n, bool form, const float2* fields_in) {
    using C = CapCfg<F>;
    Buffers& b = c->b;
    if (allow_smem(k_cap_rows<F>, C::SMEM) || allow_smem(k_cap_rows_form<F>, C::SMEM) ||
        allow_smem(k_cap_cols<F>, ColFFT<F>::SMEM))
        return TDM_ECUDA;
    if (form && n > c->chunk_cap) return TDM_EINVAL;  // the chunk buffers hold one chunk
    const size_t FF = (size_t)F * F;
    const int step = angles_per_launch(c, n);
    for (int g0 = a0; g0 < a0 + n; g0 += step) {
        const int m = a0 + n - g0 < step ? a0 + n - g0 : step;
        if (form) {
            Launch l(c, K_CAP_ROWS);
            k_cap_rows_form<F><<<dim3(F / C::B, m), C::NT, C::SMEM, c->stream>>>(
                c->p.deroul ? b.unwrapped : b.phase, b.amp, b.beta, c->p.born, b.tuk_f, c->tuk_f_flat, b.tw,
                b.fields + g0 * FF, b.r1);
        } else {
            Launch l(c, K_CAP_ROWS);
            k_cap_rows<F><<<dim3(F / C::B, m), C::NT, C::SMEM, c->stream>>>(
                fields_in ? fields_in + (g0 - a0) * FF : b.fields + g0 * FF, b.tuk_f, c->tuk_f_flat, b.tw, b.r1,
                fields_in ? b.fields + g0 * FF : nullptr);
        }
        {
            Launch l(c, K_CAP_COLS);
            using CC = ColFFT<F>;
            k_cap_cols<F><<<dim3(F / CC::B, m), CC::NT, CC::SMEM, c->stream>>>(
                b.r1, b.posspec + g0, b.s_tab, b.s_pair, c->p, b.tw, b.rec.val + g0 * FF, b.rec.z + g0 * FF, b.err);
        }
    }
    return cudaGetLastError() == cudaSuccess ? TDM_OK : TDM_ECUDA;
}

// Download of bytes from a device buffer to host memory on the download
// stream, after the work queued so far on st.
static cudaError_t download_after(tdm_ctx* c, cudaStream_t st, cudaEvent_t ev, void* host, const void* dev,
                                  size_t bytes) {
    cudaError_t e = cudaEventRecord(ev, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->dl_stream, ev, 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, c->dl_stream);
    return e;
}

// The gather of n angles' cap records into the band spectrum.
template <int W>
int launch_gather_as(tdm_ctx* c, CapRecs rec, const int2* posspec, int n, uint32_t* cnt, uint8_t* otf, int normalize,
                     cudaStream_t st) {
    const Params& p = c->p;
    const size_t smem = GatherSmem<W>::bytes(p.band, n);
    if (allow_smem(k_gather<W>, smem)) return TDM_ECUDA;
    Launch l(c, K_GATHER, st);
    k_gather<W><<<dim3((p.xb - p.xa) / W, p.yb - p.ya), W * 32, smem, st>>>(rec.val, rec.z, posspec, n, p, c->b.vol,
                                                                            cnt, otf, normalize);
    return TDM_OK;
}
int launch_gather(tdm_ctx* c, CapRecs rec, const int2* posspec, int n, uint32_t* cnt, uint8_t* otf, int normalize,
                  cudaStream_t st) {
    switch (gather_columns(c->p.D, c->p.band, n, cnt != nullptr)) {
        case 16: return launch_gather_as<16>(c, rec, posspec, n, cnt, otf, normalize, st);
        case 8: return launch_gather_as<8>(c, rec, posspec, n, cnt, otf, normalize, st);
        default: return TDM_EUNSUPPORTED;
    }
}

// x and y passes on the band planes, after the gather (DIR +1).
template <int D>
int launch_xy(tdm_ctx* c, cudaStream_t st) {
    using R = RowPass<D>;
    using P = ColPass<D>;
    const Params& p = c->p;
    if (allow_smem(k_xpass<D, 1>, R::SMEM) || allow_smem(k_ypass<D, 1>, P::SMEM)) return TDM_ECUDA;
    {
        Launch l(c, K_XPASS, st);
        k_xpass<D, 1><<<(p.band * (p.yb - p.ya) + R::B - 1) / R::B, R::NT, R::SMEM, st>>>(c->b.vol, c->b.tw, p);
    }
    {
        Launch l(c, K_YPASS, st);
        k_ypass<D, 1><<<dim3(D / P::B, p.band), P::NT, P::SMEM, st>>>(c->b.vol, c->b.tw, p);
    }
    return TDM_OK;
}

template <int D>
int volume_impl(tdm_ctx* c, int n, const VolumeOut& out, cudaStream_t st, CapRecs rec, const int2* posspec,
                cudaEvent_t ev_gathered) {
    float* re = out.re;
    float* im = out.im;
    uint8_t* otf = out.otf;
    uint32_t* cnt = out.cnt;
    using P = ColPass<D>;
    Buffers& b = c->b;
    const Params& p = c->p;
    if (allow_smem(k_zpass<D>, P::SMEM)) return TDM_ECUDA;
    // A staged output part may still be downloading from the previous volume:
    // each part's writer waits for that part's download (ev_dl) just before it runs.
    auto staged_free = [&](int part) { return cudaStreamWaitEvent(st, c->ev_dl[part], 0); };
    auto downloaded = [&](int part) { return cudaEventRecord(c->ev_dl[part], c->dl_stream); };
    if (out.host_cnt && staged_free(kOutVolumes)) return TDM_ECUDA;
    if (out.host_otf && staged_free(kOutVolumes + 1)) return TDM_ECUDA;
    // cells outside the cap band and outside the columns that caps reach carry no hits and no OTF support
    const size_t plane = (size_t)D * D, NT = (size_t)D * D * D;
    const bool all = p.xa == 0 && p.xb == D && p.ya == 0 && p.yb == D;
    const size_t lo = all ? (size_t)p.zmin * plane : NT, hi = (size_t)(p.zmin + p.band) * plane;
    if (cnt) {
        cudaMemsetAsync(cnt, 0, lo * sizeof(uint32_t), st);
        if (all) cudaMemsetAsync(cnt + hi, 0, (NT - hi) * sizeof(uint32_t), st);
    }
    if (otf) {
        cudaMemsetAsync(otf, 0, lo, st);
        if (all) cudaMemsetAsync(otf + hi, 0, NT - hi, st);
    }
    cudaEventRecord(c->ev_stage[4], st);
    if (int rc = launch_gather(c, rec, posspec, n, cnt, otf, 1, st)) return rc;
    cudaEventRecord(c->ev_stage[5], st);
    if (ev_gathered && cudaEventRecord(ev_gathered, st)) return TDM_ECUDA;
    if (out.host_cnt) {
        if (download_after(c, st, c->ev_out[kOutVolumes], out.host_cnt, cnt, NT * sizeof(uint32_t)) ||
            downloaded(kOutVolumes))
            return TDM_ECUDA;
    }
    if (out.host_otf) {
        if (download_after(c, st, c->ev_out[kOutVolumes + 1], out.host_otf, otf, NT) || downloaded(kOutVolumes + 1))
            return TDM_ECUDA;
    }
    if (int rc = launch_xy<D>(c, st)) return rc;
    // Two volumes for the host take a z pass each: the second runs while the first
    // is downloaded, and the next call's first while this call's second is.  Whole
    // volumes, because the link carries uploads and downloads at once at its full
    // rate only in contiguous copies (600 x 1024^2 to 512^3 from and to the host,
    // uploads overlapping: 131.6 volumes/s; one z pass for both by slabs of rows, whose
    // download is strided, 116).
    const bool host_vol = out.host_re || out.host_im, split = out.host_re && out.host_im;
    if (host_vol && !split && (staged_free(0) || staged_free(1))) return TDM_ECUDA;
    for (int part = 0; part < (split ? 2 : 1); ++part) {
        if (split && staged_free(part)) return TDM_ECUDA;
        {
            Launch l(c, K_ZPASS, st);
            k_zpass<D><<<dim3(D / P::B, D), P::NT, P::SMEM, st>>>(b.vol, b.tw, p, p.out_scale,
                                                                 split && part ? nullptr : re,
                                                                 split && !part ? nullptr : im);
        }
        if (host_vol) {
            const int q = part || !out.host_re;  // the volume that goes to the host
            if (download_after(c, st, c->ev_out[q], q ? out.host_im : out.host_re, q ? im : re, NT * sizeof(float)) ||
                downloaded(q))
                return TDM_ECUDA;
        }
    }
    cudaEventRecord(c->ev_stage[6], st);
    return cudaGetLastError() == cudaSuccess ? TDM_OK : TDM_ECUDA;
}

template <int D>
int forward_impl(tdm_ctx* c, const float* xn, const float* xk, int n, float2* caps, const float2* data, CapRecs res,
                 double* misfit) {
    using P = ColPass<D>;
    using R = RowPass<D>;
    Buffers& b = c->b;
    const Params& p = c->p;
    if (allow_smem(k_fzpass<D>, P::SMEM) || allow_smem(k_ypass<D, -1>, P::SMEM) || allow_smem(k_xpass<D, -1>, R::SMEM))
        return TDM_ECUDA;
    const float scale = (float)(1.0 / ((double)p.out_scale * (double)D * D * D));
    {
        Launch l(c, K_ZPASS);
        k_fzpass<D><<<dim3(D / P::B, D), P::NT, P::SMEM, c->stream>>>(xn, xk, b.tw, p, scale, b.vol);
    }
    {
        Launch l(c, K_YPASS);
        k_ypass<D, -1><<<dim3(D / P::B, p.band), P::NT, P::SMEM, c->stream>>>(b.vol, b.tw, p);
    }
    {
        Launch l(c, K_XPASS);
        k_xpass<D, -1><<<(p.band * (p.yb - p.ya) + R::B - 1) / R::B, R::NT, R::SMEM, c->stream>>>(b.vol, b.tw, p);
    }
    {
        Launch l(c, K_CAP_COLS);
        const int per = (p.F * p.F + 255) / 256;
        k_cap_sample<<<dim3(per < 16 ? per : 16, n), 256, 0, c->stream>>>(b.vol, b.posspec, p, b.s_tab, b.s_pair, data,
                                                                          caps, res.val, res.z, misfit, b.err);
    }
    return cudaGetLastError() == cudaSuccess ? TDM_OK : TDM_ECUDA;
}

template <int D>
int adjoint_impl(tdm_ctx* c, CapRecs recs, int n, float* xn, float* xk, bool normalize) {
    using P = ColPass<D>;
    Buffers& b = c->b;
    const Params& p = c->p;
    if (allow_smem(k_zpass<D>, P::SMEM)) return TDM_ECUDA;
    if (int rc = launch_gather(c, recs, b.posspec, n, nullptr, nullptr, normalize ? 1 : 0, c->stream)) return rc;
    if (int rc = launch_xy<D>(c, c->stream)) return rc;
    const float scale = normalize ? p.out_scale : (float)(1.0 / ((double)p.out_scale * (double)D * D * D));
    {
        Launch l(c, K_ZPASS);
        k_zpass<D><<<dim3(D / P::B, D), P::NT, P::SMEM, c->stream>>>(b.vol, b.tw, p, scale, xn, xk);
    }
    return cudaGetLastError() == cudaSuccess ? TDM_OK : TDM_ECUDA;
}

}  // namespace

int launch_cap(tdm_ctx* c, int a0, int n, bool form, const float2* fields_in) {
    if (c->p.F & (c->p.F - 1)) return launch_cap_generic(c, a0, n, form, fields_in);
    switch (c->p.F) {
        case 64: return cap_impl<64>(c, a0, n, form, fields_in);
        case 128: return cap_impl<128>(c, a0, n, form, fields_in);
        case 256: return cap_impl<256>(c, a0, n, form, fields_in);
        case 512: return cap_impl<512>(c, a0, n, form, fields_in);
        default: return TDM_EUNSUPPORTED;
    }
}

int launch_volume(tdm_ctx* c, int n, const VolumeOut& out, cudaStream_t st, CapRecs rec, const int2* posspec,
                  cudaEvent_t ev_gathered) {
    switch (c->p.D) {
        case 128: return volume_impl<128>(c, n, out, st, rec, posspec, ev_gathered);
        case 256: return volume_impl<256>(c, n, out, st, rec, posspec, ev_gathered);
        case 512: return volume_impl<512>(c, n, out, st, rec, posspec, ev_gathered);
        case 1024: return volume_impl<1024>(c, n, out, st, rec, posspec, ev_gathered);
        default: return TDM_EUNSUPPORTED;
    }
}

int launch_forward(tdm_ctx* c, const float* xn, const float* xk, int n, float2* caps, const float2* data,
                   CapRecs res, double* misfit) {
    switch (c->p.D) {
        case 128: return forward_impl<128>(c, xn, xk, n, caps, data, res, misfit);
        case 256: return forward_impl<256>(c, xn, xk, n, caps, data, res, misfit);
        case 512: return forward_impl<512>(c, xn, xk, n, caps, data, res, misfit);
        case 1024: return forward_impl<1024>(c, xn, xk, n, caps, data, res, misfit);
        default: return TDM_EUNSUPPORTED;
    }
}

int launch_adjoint(tdm_ctx* c, CapRecs recs, int n, float* xn, float* xk, bool normalize) {
    switch (c->p.D) {
        case 128: return adjoint_impl<128>(c, recs, n, xn, xk, normalize);
        case 256: return adjoint_impl<256>(c, recs, n, xn, xk, normalize);
        case 512: return adjoint_impl<512>(c, recs, n, xn, xk, normalize);
        case 1024: return adjoint_impl<1024>(c, recs, n, xn, xk, normalize);
        default: return TDM_EUNSUPPORTED;
    }
}

int launch_cap_pack(tdm_ctx* c, const float2* caps, int n, CapRecs recs) {
    const int per = (c->p.F * c->p.F + 255) / 256;
    {
        Launch l(c, K_CAP_COLS);
        k_cap_pack<<<dim3(per < 16 ? per : 16, n), 256, 0, c->stream>>>(caps, c->b.posspec, c->p, c->b.s_tab,
                                                                        c->b.s_pair, recs.val, recs.z, c->b.err);
    }
    return cudaGetLastError() == cudaSuccess ? TDM_OK : TDM_ECUDA;
}

int launch_tv_step(tdm_ctx* c, const float* xn, const float* xk, const float* gn, const float* gk, float step,
                   float tv_n, float tv_k, float eps, float nlo, float nhi, float klo, float khi, float* xn_out,
                   float* xk_out) {
    const int D = c->p.D;
    {
        Launch l(c, K_FORM);
        const TvChannel cn{xn, gn, xn_out, tv_n, nlo, nhi}, ck{xk, gk, xk_out, tv_k, klo, khi};
        k_tv_step<<<dim3((unsigned)((size_t)D * D * D / (1024 * kTvPlanes)), xk ? 2 : 1), 256, 0, c->stream>>>(cn, ck, ilog2c(D),
                                                                                                 step, eps * eps);
    }
    return cudaGetLastError() == cudaSuccess ? TDM_OK : TDM_ECUDA;
}

}  // namespace tdm
