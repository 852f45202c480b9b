// Herraez phase unwrapping (VOLKOV 0): phaseUnwrapping_Mat,
// pretraitement_hors_axe_CPU/deroulement_herraez.cpp:32-74, as
// pretraitement_hors_axe_CPU/main.cpp:262-266 calls it on each angle's wrapped
// phase.  The result is the reference's bit for bit, given the same float
// wrapped phase:
//
//  k_hz_reliability  initialisePIXELs and calculate_reliability (:333-413):
//                    second differences of the wrapped phase in float for the
//                    interior; border pixels keep 9999999 + rand() (an int sum
//                    that wraps past INT_MAX), from the C library's generator
//                    as the reference's loop draws it: F^2 draws per earlier
//                    angle (host table, crand_border_table).
//  k_hz_sort_base    horizentalEDGEs, verticalEDGEs (:415-459): each edge's
//                    reliability (the two pixels' sum) and its 2 pi jump, and
//                    the deep levels of quick_sort (:163-213): the reference's
//                    merge sort on edge indices, which halves with size/2 so
//                    that the last index of an odd-sized run stays where it
//                    is; the later merges then see runs that are not sorted.
//                    Mix (:113-159) merges them by comparing heads, which
//                    interleaves two runs as a stable merge of their prefix
//                    maxima does, so each element carries its run's prefix
//                    maximum: merging leaves it unchanged, and an odd node's
//                    leftover takes the maximum of its node when it joins its
//                    parent's run.  Every node of a depth has the same size;
//                    a CTA sorts one node of at most kSortBase edges in shared
//                    memory, where each element of a node's two halves finds
//                    its place by a binary search on the other half's prefix
//                    maxima (ties: the first half first, as in Mix).
//  k_hz_merge        the levels above, one launch each: a CTA writes kSortBase
//                    elements of a node's merged run, whose sources it finds
//                    by a search along the merge's diagonal.
//  k_hz_gather       gatherPIXELs and unwrapImage (:461-575), one CTA per
//                    angle: the edges in sorted order merge pixel groups.
//                    The reference keeps each group as a linked list and adds
//                    the merged group's 2 pi offset to every member; here the
//                    groups are a union-find forest in shared memory whose
//                    links carry the 2 pi offset to the parent (int8; -128
//                    marks a root, whose parent slot holds the group's size),
//                    and which takes the same decisions (a lone pixel 2 joins
//                    pixel 1's group, else a lone pixel 1 joins pixel 2's,
//                    else the larger group absorbs the other, ties to group
//                    2), so each pixel's count is the reference's.  The merges
//                    run many at a time, each only when it is certain to be
//                    the one that the sorted order makes (see the kernel).
#include <type_traits>

#include "tdm_internal.cuh"

namespace tdm {
namespace {

constexpr float kHzPi = 3.141592654f, kHzTwoPi = 6.283185307f;  // deroulement_herraez.cpp:9-10
constexpr int kHzThreads = 256;

__device__ __forceinline__ float hz_wrap(float v) {  // wrap (:357-365)
    return v > kHzPi ? __fsub_rn(v, kHzTwoPi) : (v < -kHzPi ? __fadd_rn(v, kHzTwoPi) : v);
}

// Pixels of edge e: the F (F - 1) horizontal edges row by row, then the
// (F - 1) F vertical ones.
__device__ __forceinline__ void hz_edge(int e, int F, int& p1, int& p2) {
    const int nh = F * (F - 1);
    if (e < nh) {
        const int i = e / (F - 1);
        p1 = e + i;
        p2 = p1 + 1;
    } else {
        p1 = e - nh;
        p2 = p1 + F;
    }
}

// An edge's payload through the sort: its first pixel, whether it is
// vertical, and its 2 pi jump + 1: (p1 << 3) | (vertical << 2) | (jump + 1).
__device__ __forceinline__ void hz_payload_pixels(uint32_t pl, int F, int& p1, int& p2) {
    p1 = (int)(pl >> 3);
    p2 = p1 + ((pl & 4u) ? F : 1);
}

__global__ void __launch_bounds__(kHzThreads)
k_hz_reliability(const float* __restrict__ phase, const int* __restrict__ border_rand, int a0, int F,
                 float* __restrict__ rel) {
    const int a = blockIdx.y, FF = F * F;
    const int p = blockIdx.x * kHzThreads + threadIdx.x;
    if (p >= FF) return;
    const float* ph = phase + (size_t)a * FF;
    const int i = p / F, j = p - i * F;
    float r;
    if (i == 0 || j == 0 || i == F - 1 || j == F - 1) {
        // border index: row 0, then columns 0 and F - 1 of rows 1 .. F - 2, then row F - 1
        const int b = i == 0 ? j : (i == F - 1 ? F + 2 * (F - 2) + j : F + 2 * (i - 1) + (j ? 1 : 0));
        const uint32_t v = 9999999u + (uint32_t)border_rand[(size_t)(a0 + a) * (4 * F - 4) + b];
        r = __int2float_rn((int)v);
    } else {
        const float c = ph[p];
        auto d2 = [&](int o) { return __fsub_rn(hz_wrap(__fsub_rn(ph[p - o], c)), hz_wrap(__fsub_rn(c, ph[p + o]))); };
        const float H = d2(1), V = d2(F), D1 = d2(F + 1), D2 = d2(F - 1);
        r = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(H, H), __fmul_rn(V, V)), __fmul_rn(D1, D1)), __fmul_rn(D2, D2));
    }
    rel[(size_t)a * FF + p] = r;
}

// Sort arrays of one angle: the keys (each element's run prefix maximum)
// and the payloads, ne each.  The chunk's angle i keeps its arrays at offset
// i * stride.
struct SortBuf {
    float* eff;
    uint32_t* pay;
};

// Elements a CTA sorts or merges: keys and payloads twice take 32 KB of shared
// memory (several CTAs an SM), and 256 threads take 8 each.
constexpr int kSortBase = 2048;
constexpr int kSortPer = kSortBase / kHzThreads;

// Start of node `id` (path bits, first halving in the highest) of depth
// `depth` of the sort of n elements; n becomes the node's size.
__device__ __forceinline__ int hz_node(int id, int depth, int& n) {
    int s = 0;
    for (int d = depth - 1; d >= 0; --d) {
        n /= 2;
        if ((id >> d) & 1) s += n;
    }
    return s;
}

// CTA x < 2^depth: the edges of node x of that depth (at most kSortBase),
// sorted as the reference's recursion below that node leaves them, into out.
// The last CTA: the leftovers of the odd nodes above, which stay in place
// until their own node is merged, into both buffers.
__global__ void __launch_bounds__(kHzThreads)
k_hz_sort_base(const float* __restrict__ phase, const float* __restrict__ rel, int F, size_t stride, int depth,
               SortBuf out, SortBuf other) {
    __shared__ float keys[2][kSortBase];
    __shared__ uint32_t pays[2][kSortBase];
    const int a = blockIdx.y, FF = F * F, ne = 2 * F * (F - 1);
    const size_t base = a * stride;
    const float* ph = phase + (size_t)a * FF;
    const float* rl = rel + (size_t)a * FF;
    auto edge = [&](int e, float& key, uint32_t& pay) {
        int p1, p2;
        hz_edge(e, F, p1, p2);
        const float d = __fsub_rn(ph[p1], ph[p2]);  // find_wrap (:368-380)
        const int jump = d > kHzPi ? -1 : (d < -kHzPi ? 1 : 0);
        key = __fadd_rn(rl[p1], rl[p2]);  // a run of one
        pay = ((uint32_t)p1 << 3) | (p2 - p1 == 1 ? 0u : 4u) | (uint32_t)(jump + 1);
    };
    if (blockIdx.x == (1u << depth)) {
        for (int t = threadIdx.x; t < (1 << depth) - 1; t += kHzThreads) {
            const int d = 31 - __clz(t + 1), id = t + 1 - (1 << d);  // node id of depth d
            int n = ne;
            const int s = hz_node(id, d, n);
            if (n & 1) {
                float key;
                uint32_t pay;
                edge(s + n - 1, key, pay);
                out.eff[base + s + n - 1] = other.eff[base + s + n - 1] = key;
                out.pay[base + s + n - 1] = other.pay[base + s + n - 1] = pay;
            }
        }
        return;
    }
    int n0 = ne;
    const int s0 = hz_node(blockIdx.x, depth, n0);
    for (int i = threadIdx.x; i < n0; i += kHzThreads) {
        edge(s0 + i, keys[0][i], pays[0][i]);
        // with NaN keys two elements can claim one place: the place left over then still names an edge
        pays[1][i] = pays[0][i];
    }
    __syncthreads();
    int levels = 0;  // depths below this node whose nodes have at least 2 elements
    for (int n = n0; n >= 2; n /= 2) ++levels;
    int cur = 0;
    for (int lv = levels - 1; lv >= 0; --lv, cur ^= 1) {
        const float* k = keys[cur];
        for (int i = threadIdx.x; i < n0; i += kHzThreads) {
            int s = 0, n = n0;
            bool inside = true;
            for (int d = 0; d < lv; ++d) {
                const int h = n / 2;
                if (i >= s + 2 * h) {
                    inside = false;  // the leftover of an odd-sized ancestor
                    break;
                }
                if (i >= s + h) s += h;
                n = h;
            }
            float x = k[i];
            int dst = i;
            const int h = n / 2;
            if (inside && i < s + 2 * h) {
                const bool first = i < s + h;
                const int o = first ? s + h : s;  // the other half
                int lo = 0, hi = h;
                while (lo < hi) {  // elements of the other half that come before x
                    const int m = (lo + hi) >> 1;
                    const float v = k[o + m];
                    if (first ? v < x : v <= x) lo = m + 1;
                    else hi = m;
                }
                dst = (first ? i : i - h) + lo;
            } else if (inside) {  // the odd node's leftover joins the node's run at its end
                x = fmaxf(fmaxf(k[s + h - 1], k[s + 2 * h - 1]), x);
            }
            keys[cur ^ 1][dst] = x;
            pays[cur ^ 1][dst] = pays[cur][i];
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n0; i += kHzThreads) {
        out.eff[base + s0 + i] = keys[cur][i];
        out.pay[base + s0 + i] = pays[cur][i];
    }
}

// How many of the first `diag` elements of the merge of A and B (h each,
// nondecreasing; ties: A first) come from A; the warp's lanes probe 32 places a step.
__device__ __forceinline__ int hz_diagonal(const float* A, const float* B, int h, int diag) {
    const int lane = threadIdx.x & 31;
    int lo = max(0, diag - h), hi = min(diag, h);
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32, m = lo + lane * step;
        const bool p = m < hi && A[m] <= B[diag - 1 - m];  // true up to the answer
        const int c = __popc(__ballot_sync(0xffffffffu, p));
        if (c == 0) return lo;
        hi = min(hi, lo + c * step);
        lo += (c - 1) * step + 1;
    }
    return lo;
}

// Depth `depth` of the sort: CTA x merges piece x % pieces (kSortBase elements)
// of the halves of node x / pieces; an odd node's leftover joins its run.
__global__ void __launch_bounds__(kHzThreads)
k_hz_merge(SortBuf in, SortBuf out, size_t stride, int ne, int depth, int pieces) {
    __shared__ float key[kSortBase];
    __shared__ uint32_t pay[kSortBase];
    __shared__ int s_from[2];
    const size_t base = blockIdx.y * stride;
    int n = ne;
    const int s = hz_node(blockIdx.x / pieces, depth, n), h = n / 2;
    const float *A = in.eff + base + s, *B = A + h;
    const uint32_t *PA = in.pay + base + s, *PB = PA + h;
    const int d0 = (int)(blockIdx.x % pieces) * kSortBase, d1 = min(d0 + kSortBase, 2 * h);
    const int w = threadIdx.x >> 5;
    if (w < 2) {
        const int r = hz_diagonal(A, B, h, w ? d1 : d0);
        if ((threadIdx.x & 31) == 0) s_from[w] = r;
    }
    __syncthreads();
    // (clamped: with NaN keys the two searches need not agree)
    const int i0 = s_from[0], na = min(max(s_from[1] - i0, 0), d1 - d0), j0 = d0 - i0, nb = d1 - d0 - na;
    for (int t = threadIdx.x; t < na + nb; t += kHzThreads) {
        key[t] = t < na ? A[i0 + t] : B[j0 + t - na];
        pay[t] = t < na ? PA[i0 + t] : PB[j0 + t - na];
    }
    __syncthreads();
    // each thread: kSortPer consecutive outputs
    const int o0 = threadIdx.x * kSortPer, o1 = min(o0 + kSortPer, na + nb);
    float rk[kSortPer];
    uint32_t rp[kSortPer];
    if (o0 < o1) {
        int lo = max(0, o0 - nb), hi = min(o0, na);
        while (lo < hi) {
            const int m = (lo + hi) >> 1;
            if (key[m] <= key[na + o0 - 1 - m]) lo = m + 1;
            else hi = m;
        }
        int i = lo, j = o0 - lo;
#pragma unroll
        for (int t = 0; t < kSortPer; ++t) {
            if (o0 + t < o1) {
                const bool a = j >= nb || (i < na && key[i] <= key[na + j]);
                const int f = a ? i++ : na + j++;
                rk[t] = key[f];
                rp[t] = pay[f];
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kSortPer; ++t)
        if (o0 + t < o1) {
            key[o0 + t] = rk[t];
            pay[o0 + t] = rp[t];
        }
    __syncthreads();
    for (int t = threadIdx.x; t < na + nb; t += kHzThreads) {
        out.eff[base + s + d0 + t] = key[t];
        out.pay[base + s + d0 + t] = pay[t];
    }
    if (d0 == 0 && threadIdx.x == 0 && (n & 1)) {
        const size_t o = base + s + n - 1;
        out.eff[o] = fmaxf(fmaxf(A[h - 1], B[h - 1]), in.eff[o]);
        out.pay[o] = in.pay[o];
    }
}

// The forest of k_hz_gather for F x F pixels: per pixel the parent (or, at a
// root, the group's size - 1) and the 2 pi offset to the parent as int8,
// kHzRoot marking a root.  In shared memory (uint16 parents) up to 256^2
// pixels: 3 bytes a pixel, beside the three tables of the merging.
constexpr int kHzRoot = -128;
constexpr int kGatherThreads = 256;
constexpr int kHzBuckets = 2048;  // three tables and the ring beside the forest of 256^2 pixels: 225 KB
constexpr int kHzRing = 4 * kGatherThreads;
size_t hz_gather_smem(int F, bool shared) {
    const size_t n = (size_t)F * F;
    return (3 * kHzBuckets + kHzRing) * sizeof(uint32_t) + (shared ? n * 3 : 0);
}

// Forest in shared memory (up to 256^2 pixels) or in global memory (32-bit
// parents, n of them and then n offsets, one CTA's own).
struct SharedForest {
    uint32_t* up;  // two parents a word
    int8_t* pot;
    __device__ int parent(int p) const { return reinterpret_cast<const uint16_t*>(up)[p]; }
    __device__ int offset(int p) const { return pot[p]; }
    // root c of size sc goes under parent r (which gains sc pixels) with offset v.  Other threads change the
    // other halves of the two words at the same time, so both changes are atomic.
    __device__ void link(int c, int sc, int r, int v) {
        atomicXor(&up[c >> 1], (uint32_t)((sc - 1) ^ r) << (16 * (c & 1)));
        atomicAdd(&up[r >> 1], (uint32_t)sc << (16 * (r & 1)));
        pot[c] = (int8_t)v;
    }
    __device__ void publish() const {}
};
struct GlobalForest {
    uint32_t* up;
    int8_t* pot;
    __device__ int parent(int p) const { return *reinterpret_cast<volatile uint32_t*>(&up[p]); }
    __device__ int offset(int p) const { return *reinterpret_cast<volatile int8_t*>(&pot[p]); }
    __device__ void link(int c, int sc, int r, int v) {
        *reinterpret_cast<volatile uint32_t*>(&up[c]) = (uint32_t)r;
        atomicAdd(&up[r], (uint32_t)sc);
        *reinterpret_cast<volatile int8_t*>(&pot[c]) = (int8_t)v;
    }
    __device__ void publish() const { __threadfence(); }  // before the barrier that other threads read after
};

// One CTA per angle merges the groups of the sorted edges.  One edge after the
// other is a chain of shared-memory loads (about 380 cycles an edge: 23 ms for
// 256^2 pixels); instead each thread holds one pending edge, taken in sorted
// order, and rounds of four steps make every merge that is certain to be the
// sorted order's, many at once.  Hash tables of roots hold edges' places in
// the order; roots that share an entry only wait longer.
//   1. The edge's two roots (walking on from the roots it knew) and their
//      sizes; an edge within one group is done.  By the sizes, one root (the
//      small one) would go under the other (the big one).  first: the first
//      pending edge at each root.
//   2. An edge that is the first at its small root is settled: no earlier edge
//      can change that group any more, and the decision holds however much
//      the big group grows meanwhile.  second: the first of the other edges at
//      each root.  bar: the first edge at each root that might do other than
//      put a settled group under it: the edges whose small root it is, and at
//      their big root the edges that are not settled.
//   3. A settled edge brings its small group's other edges to the big root:
//      bar takes second of the small root there.
//   4. A settled edge that nothing bars at its big root merges: whatever
//      earlier edges do there, they put smaller groups under it, in any order.
//      A group of more than half of the pixels takes in every other group it
//      meets, so at such a big root nothing bars, and nothing is noted.
// So a large group takes in many settled neighbours at once, and the first
// pending edge always merges, so the rounds end.  The offset of the edge's two
// groups, c = count(pixel 1) - jump - count(pixel 2) relative to their roots,
// is kept up as the roots change.
// 48 angles of 256^2 as chunks of 16, with the sort: 70.5 -> 7.6 ms (128 threads
// 7.8, 512 8.7, 1024 more: fewer rounds, but each issues more).
template <class Forest>
__global__ void __launch_bounds__(kGatherThreads)
k_hz_gather(const uint32_t* __restrict__ pays, size_t stride, const float* __restrict__ phase, int F,
            float* __restrict__ unwrapped, int* __restrict__ err, unsigned char* __restrict__ forest,
            size_t forest_stride) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int s_free[32];
    const int a = blockIdx.x, n = F * F, ne = 2 * F * (F - 1);
    uint32_t* first = reinterpret_cast<uint32_t*>(smraw);
    uint32_t *second = first + kHzBuckets, *bar = second + kHzBuckets, *ring = bar + kHzBuckets;
    constexpr bool SHARED = std::is_same<Forest, SharedForest>::value;
    Forest f;
    f.up = SHARED ? ring + kHzRing : reinterpret_cast<uint32_t*>(forest + a * forest_stride);
    f.pot = reinterpret_cast<int8_t*>(SHARED ? f.up + n / 2 : f.up + n);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int p = tid; p < (SHARED ? n / 2 : n); p += kGatherThreads) f.up[p] = 0;  // roots of groups of size 1
    for (int p = tid; p < n / 4; p += kGatherThreads) reinterpret_cast<uint32_t*>(f.pot)[p] = 0x80808080u;
    f.publish();
    // table values carry the round in their upper bits, later rounds smaller, so that they need clearing
    // only every kRounds rounds; an edge's place in the sorted order fits the lower 20 bits
    constexpr int kRounds = 4095;
    const uint32_t* ps = pays + a * stride;
    auto bucket = [](int r) { return ((uint32_t)r * 2654435761u) >> 21; };
    static_assert(kHzBuckets == 2048, "11 bits of hash");
    // a table entry's minimum; at a big root most threads find a smaller value there already, and atomics on
    // one address run one after the other
    auto lower = [](uint32_t* table, uint32_t at, uint32_t key) {
        if (*reinterpret_cast<volatile uint32_t*>(&table[at]) > key) atomicMin(&table[at], key);
    };
    // sorted edges wait in a ring, loaded a round ahead of their use
    int loaded = 0;
    for (; loaded < kHzRing / 2; loaded += kGatherThreads)
        if (loaded + tid < ne) ring[loaded + tid] = ps[loaded + tid];
    bool have = false;
    int next = 0, r1 = 0, r2 = 0, c = 0, bad = 0;
    uint32_t k = 0;
    for (int round = 0;; ++round) {
        if (round % kRounds == 0) {
            __syncthreads();  // the last round's reads of the tables
            for (int i = tid; i < 3 * kHzBuckets; i += kGatherThreads) first[i] = 0xffffffffu;
        }
        // new edges for the threads without one
        const unsigned fb = __ballot_sync(0xffffffffu, !have);
        if (lane == 0) s_free[w] = __popc(fb);
        __syncthreads();
        const int fr = lane < kGatherThreads / 32 ? s_free[lane] : 0;
        int incl = fr;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        if (total == kGatherThreads && next >= ne) break;  // no edge pending, none left
        const int mine = next + __shfl_sync(0xffffffffu, incl - fr, w) + __popc(fb & ((1u << lane) - 1u));
        if (!have && mine < ne) {
            const uint32_t pl = ring[mine % kHzRing];
            k = (uint32_t)mine;
            c = 1 - (int)(pl & 3u);
            hz_payload_pixels(pl, F, r1, r2);
            have = true;
        }
        next = min(ne, next + total);
        const bool fill = loaded < ne && loaded - next < kHzRing / 2;  // stored below, after a barrier
        const uint32_t ahead = fill && loaded + tid < ne ? ps[loaded + tid] : 0;
        const uint32_t key = ((uint32_t)(kRounds - 1 - round % kRounds) << 20) | k;
        // 1. roots and sizes
        int small = 0, big = 0, ssz = 0, v = 0;
        uint32_t hs = 0, hb = 0;
        bool hub = false;
        if (have) {
            int o1 = f.offset(r1), u1 = f.parent(r1), o2 = f.offset(r2), u2 = f.parent(r2);
            while (o1 != kHzRoot || o2 != kHzRoot) {  // both walks at once, a link's two halves at once
                if (o1 != kHzRoot) c += o1, r1 = u1;
                if (o2 != kHzRoot) c -= o2, r2 = u2;
                o1 = f.offset(r1), u1 = f.parent(r1), o2 = f.offset(r2), u2 = f.parent(r2);
            }
            have = r1 != r2;
            const int s1 = u1 + 1, s2 = u2 + 1;
            const bool two = s2 == 1 || (s1 != 1 && s1 > s2);  // pixel 2's group goes under pixel 1's
            small = two ? r2 : r1, big = two ? r1 : r2, ssz = two ? s2 : s1, v = two ? c : -c;
            hub = (two ? s1 : s2) > n / 2;
            hs = bucket(small), hb = bucket(big);
            if (have) {
                atomicMin(&first[hs], key);
                if (!hub) lower(first, hb, key);
            }
        }
        __syncthreads();
        // 2. settled edges, the roots' other edges, and what bars merges
        bool settled = false;
        if (have) {
            settled = first[hs] == key;
            const bool other = first[hb] != key;
            if (!settled) atomicMin(&second[hs], key);
            atomicMin(&bar[hs], key);
            if (!hub) {
                if (other) lower(second, hb, key);
                if (!settled) lower(bar, hb, key);
            }
        }
        __syncthreads();
        // 3. (a second of an earlier round is above every key of this one)
        if (settled && !hub) lower(bar, hb, second[hs]);
        __syncthreads();
        // 4. merges
        if (settled && (hub || key <= bar[hb])) {
            const bool over = v < -127 || v > 127;
            bad |= over;
            f.link(small, ssz, big, over ? 0 : v);
            have = false;
        }
        if (fill) {
            if (loaded + tid < ne) ring[(loaded + tid) % kHzRing] = ahead;
            loaded += kGatherThreads;
        }
        f.publish();
    }
    if (bad) atomicOr(err, 8);
    const float* ph = phase + (size_t)a * n;
    float* out = unwrapped + (size_t)a * n;
    for (int p = tid; p < n; p += kGatherThreads) {
        int acc = 0;
        int q = p;
        for (int o; (o = f.offset(q)) != kHzRoot; q = f.parent(q)) acc += o;
        out[p] = __fadd_rn(ph[p], __fmul_rn(kHzTwoPi, __int2float_rn(acc)));
    }
}

}  // namespace

// The m angles of the chunk starting at stack angle a0: b.phase -> b.unwrapped,
// with b.gx (reliabilities) and b.qc / b.tq (keys and payloads, ping-pong) as
// scratch.
int launch_herraez(tdm_ctx* c, int a0, int m) {
    Buffers& b = c->b;
    const int F = c->p.F, FF = F * F, ne = 2 * F * (F - 1);
    const size_t stride = (size_t)c->p.L * F * 2;  // floats per angle in qc and tq (L F complex >= 2 ne)
    SortBuf buf[2];
    float* base[2] = {reinterpret_cast<float*>(b.qc), reinterpret_cast<float*>(b.tq)};
    for (int k = 0; k < 2; ++k) buf[k] = SortBuf{base[k], reinterpret_cast<uint32_t*>(base[k] + ne)};
    const bool shared = F <= 256;  // uint16 parents
    const size_t smem = hz_gather_smem(F, shared);
    if (!b.hz_rand || smem > kMaxSmemPerCta) return TDM_EUNSUPPORTED;
    const void* gather = shared ? reinterpret_cast<const void*>(k_hz_gather<SharedForest>)
                                : reinterpret_cast<const void*>(k_hz_gather<GlobalForest>);
    if (max_dynamic_smem(gather, smem) != cudaSuccess) return TDM_ECUDA;
    {
        Launch l(c, K_HERRAEZ);
        k_hz_reliability<<<dim3((FF + kHzThreads - 1) / kHzThreads, m), kHzThreads, 0, c->stream>>>(
            b.phase, b.hz_rand, a0, F, b.gx);
    }
    int depth = 0;  // the first depth whose nodes fit one CTA
    while ((ne >> depth) > kSortBase) ++depth;
    {
        Launch l(c, K_HERRAEZ);
        k_hz_sort_base<<<dim3((1 << depth) + 1, m), kHzThreads, 0, c->stream>>>(b.phase, b.gx, F, stride, depth,
                                                                                buf[0], buf[1]);
    }
    int cur = 0;
    for (int d = depth - 1; d >= 0; --d, cur ^= 1) {
        const int pieces = (2 * ((ne >> d) / 2) + kSortBase - 1) / kSortBase;
        Launch l(c, K_HERRAEZ);
        k_hz_merge<<<dim3(pieces << d, m), kHzThreads, 0, c->stream>>>(buf[cur], buf[cur ^ 1], stride, ne, d, pieces);
    }
    if (shared) {
        Launch l(c, K_HERRAEZ);
        k_hz_gather<SharedForest><<<m, kGatherThreads, smem, c->stream>>>(buf[cur].pay, stride, b.phase, F,
                                                                          b.unwrapped, b.err, nullptr, 0);
    } else {  // the forest in the other sort buffer, free now: 5 bytes a pixel within 16 F^2 an angle
        Launch l(c, K_HERRAEZ);
        k_hz_gather<GlobalForest><<<m, kGatherThreads, smem, c->stream>>>(
            buf[cur].pay, stride, b.phase, F, b.unwrapped, b.err, reinterpret_cast<unsigned char*>(base[cur ^ 1]),
            stride * sizeof(float));
    }
    return cudaGetLastError() == cudaSuccess ? TDM_OK : TDM_ECUDA;
}

}  // namespace tdm
