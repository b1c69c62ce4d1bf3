// march.cuh -- full-field passes: the fused labelling + first detection, the
// full detection sweeps and the direction codes, and the two-field pass of the
// verification; included after tiled.cuh.
//
// One block of 32 x 4 threads owns a 32 x 8 column of the field (two voxels
// per thread and plane, one above the other in y) and marches it through g.zc
// planes.  What bounds these passes is instruction issue and the ALU pipe, not
// HBM, so the design counts instructions per voxel:
//
//  * Tagged proxies.  A cell's 32-bit value in shared memory is the high 28
//    bits of its key (proxy_of) and, in the low 4 bits, the tag
//    (7x + y + 2z) mod 16 of its ABSOLUTE coordinates.  The 15 stencil points
//    have 15 different tags around any voxel ((7dx + dy + 2dz) mod 16 takes
//    every value but 8), so the packed maximum names the winning cell and no
//    chain adds a rank to its candidates.
//  * Certificates.  A second chain over the values with the tag bits flipped
//    picks, among cells that share the 28 value bits, the lowest tag instead
//    of the highest: both chains name the same cell exactly when the winner is
//    unique.  Otherwise the voxel goes to the block's exact queue.
//  * Plane blocks.  In one plane the stencil uses the 2x2 blocks
//      U = {(x,y-1), (x+1,y-1), (x,y), (x+1,y)}
//      V = {(x-1,y), (x,y), (x-1,y+1), (x,y+1)}
//    and the whole stencil of a voxel of plane z is U(z-1), U(z), V(z) and
//    V(z+1).  A thread reads the 10 cells that a plane contributes to its two
//    voxels once, keeps U and G = U(z-1) + U(z) + V(z) in registers, and
//    finishes a voxel when the next plane brings V.  The two voxels share the
//    row pairs of their blocks, so a chain takes 8 min/max and 5 shared-memory
//    loads per voxel instead of 14 (plus the rank adds) and 15.
//  * Cells outside the domain are never read: a thread on an x or y face reads
//    another cell of the same 2x2 block instead (the same value and tag twice
//    changes no winner and no certificate), and a plane outside in z
//    contributes the chains' identities.
//  * Planes arrive in a ring of raw stages several planes ahead, by TMA or by
//    cp.async, so no register holds a value in flight.
//
// Exact decisions.  A voxel whose certificate fails (ties in the truncated
// proxies) is queued in shared memory and decided on full keys, gathered from
// global memory (recently loaded, so mostly L2 hits), by the whole block: full
// warps instead of one lane per warp, no second kernel and no global list.
// The same holds for voxels whose two codes differ and that need the rules,
// and for values that may be NaN or the sentinel.  The queues are emptied when
// one could overflow in the next plane, and at the end.  Where most certificates
// of one field fail, the rest of the column needs none (march_tied).
//
// Bitmaps of a column.  A word of the request and mismatch bitmaps is one row
// of one plane of the column: collected in shared memory and written once, with
// the group flags that k_sweeps reads (atomics per voxel before: a dense 256^3
// fp32 first pass took 754 us, then 626; with the values compared directly on
// ties 485).
//
// Measured at 512^3, issue-bound throughout: first pass fp64 1.50 -> 1.14 ms
// (350 -> 220 warp instructions per 32 voxels), fp32 1.00 ms; codes alone
// 0.56 ms fp64, 0.53 ms fp32.  One voxel per thread, 256-thread blocks, the two
// fields on different warps and 15 gathers per lane in the exact queue were all
// slower.
#pragma once
#include <algorithm>
#include <limits>
#include <type_traits>

#include "tiled.cuh"

namespace pmsz {

enum MarchMode { kFirst = 0, kDetect = 1, kCodes = 2, kPair = 3 };
constexpr bool march_pair(int mode) { return mode == kFirst || mode == kPair; }  // marches two fields
constexpr bool march_edits(int mode) { return mode == kFirst || mode == kDetect; }  // asks for edits

__host__ __device__ constexpr uint32_t stencil_tag(int x, int y, int z) {
    return (7u * static_cast<uint32_t>(x) + static_cast<uint32_t>(y) + 2u * static_cast<uint32_t>(z)) & 15u;
}
// Stencil rank of a tag difference (winner - voxel) mod 16; difference 8 does
// not occur.
constexpr uint64_t tag_rank_table() {
    uint64_t t = 0;
    for (int r = 0; r < 15; ++r)
        t |= static_cast<uint64_t>(r) << (4 * stencil_tag(rank_dx(r), rank_dy(r), rank_dz(r)));
    return t;
}
constexpr bool tags_distinct() {
    uint32_t seen = 0;
    for (int r = 0; r < 15; ++r) {
        const uint32_t b = 1u << stencil_tag(rank_dx(r), rank_dy(r), rank_dz(r));
        if (seen & b) return false;
        seen |= b;
    }
    return true;
}
static_assert(tags_distinct(), "the 15 stencil points must carry 15 different tags");

__device__ __forceinline__ uint8_t tag_pair_code(uint32_t d) {  // two tag differences -> code byte
    constexpr uint64_t t = tag_rank_table();
    return static_cast<uint8_t>(((t >> (4 * (d & 15u))) & 15u) | (((t >> (4 * ((d >> 4) & 15u))) & 15u) << 4));
}

__device__ __forceinline__ uint32_t rank_pair_tags(uint32_t code) {  // and back
    constexpr uint64_t t = [] {
        uint64_t v = 0;
        for (int r = 0; r < 15; ++r) v |= static_cast<uint64_t>(stencil_tag(rank_dx(r), rank_dy(r), rank_dz(r))) << (4 * r);
        return v;
    }();
    return (static_cast<uint32_t>(t >> (4 * (code & 15u))) & 15u) | ((static_cast<uint32_t>(t >> (4 * (code >> 4))) & 15u) << 4);
}

// Maximum and minimum of a set of tagged values.
struct Ext2 {
    uint32_t hi, lo;
};
__device__ __forceinline__ Ext2 ext2(uint32_t a, uint32_t b) { return Ext2{max(a, b), min(a, b)}; }
__device__ __forceinline__ Ext2 join(const Ext2 &a, const Ext2 &b) { return Ext2{max(a.hi, b.hi), min(a.lo, b.lo)}; }
__device__ __forceinline__ Ext2 join(const Ext2 &a, const Ext2 &b, const Ext2 &c) {
    return Ext2{__vimax3_u32(a.hi, b.hi, c.hi), __vimin3_u32(a.lo, b.lo, c.lo)};
}
__device__ __forceinline__ Ext2 join(uint32_t a, uint32_t b, const Ext2 &c) {
    return Ext2{__vimax3_u32(a, b, c.hi), __vimin3_u32(a, b, c.lo)};
}

// Order-preserving signed keys: the magnitude bits, negated where the sign is set
// (-0 and +0 are both 0; the order of okey, NaN included).
__device__ __forceinline__ int32_t signed_key(float v) {
    const int32_t b = __float_as_int(v), m = b >> 31;
    return ((b & 0x7FFFFFFF) ^ m) - m;
}
__device__ __forceinline__ int64_t signed_key(double v) {
    const int64_t b = __double_as_longlong(v), m = b >> 63;
    return ((b & 0x7FFFFFFFFFFFFFFFll) ^ m) - m;
}

// Steepest ranks of one voxel on the values load(r) of its valid stencil points
// (arg_ext's rule: ties by rank).  fp32 takes all 15 at once: their extremes by
// max and min, then the last rank that holds the maximum and the first that holds
// the minimum; without NANS (a correction refuses them after its first pass, and
// only the direction codes order them) on the values themselves, NaN standing
// for a point outside the domain, -0 and +0 equal in both forms.  A first pass
// over plateaus (256^3 fp32) takes 485 us so instead of 626 on keys one by one, 311 M
// fp32 voxels with many ties 2.98 ms instead of 3.29.  fp64: LOADS keys at a time.
template <typename T, bool NANS, int LOADS, class Load>
__device__ __forceinline__ void scan_ranks(Load load, uint32_t valid, int &asc, int &desc) {
    asc = desc = kSelf;
    if constexpr (sizeof(T) == 4 && !NANS) {
        T t[15];
#pragma unroll
        for (int r = 0; r < 15; ++r) t[r] = ((valid >> r) & 1u) ? load(r) : __int_as_float(0x7FC00000);
        T hi = t[0], lo = t[0];
#pragma unroll
        for (int r = 1; r < 15; r += 2) {
            hi = fmaxf(fmaxf(hi, t[r]), t[r + 1]);
            lo = fminf(fminf(lo, t[r]), t[r + 1]);
        }
#pragma unroll
        for (int r = 0; r < 15; ++r) {
            if (t[r] == hi) asc = r;
            if (t[14 - r] == lo) desc = 14 - r;
        }
    } else {
        using K = std::conditional_t<sizeof(T) == 4, int32_t, int64_t>;
        K hi = std::numeric_limits<K>::min(), lo = std::numeric_limits<K>::max();
#pragma unroll
        for (int r0 = 0; r0 < 15; r0 += LOADS) {
            T t[LOADS];
#pragma unroll
            for (int j = 0; j < LOADS; ++j) t[j] = ((valid >> (r0 + j)) & 1u) ? load(r0 + j) : T(0);
#pragma unroll
            for (int j = 0; j < LOADS; ++j) {
                const K k = signed_key(t[j]);
                if ((valid >> (r0 + j)) & 1u) {
                    if (k >= hi) { hi = k; asc = r0 + j; }
                    if (k < lo) { lo = k; desc = r0 + j; }
                }
            }
        }
    }
}

// The same on values that lie in shared memory: all at once, as they are where no
// sign is set (their bits are in order then), else as keys.
template <typename T, class Load>
__device__ __forceinline__ void scan_tile(Load load, uint32_t valid, int &asc, int &desc) {
    using K = std::conditional_t<sizeof(T) == 4, int32_t, int64_t>;
    constexpr K kLow = std::numeric_limits<K>::min(), kHigh = std::numeric_limits<K>::max();
    K k[15], signs = 0;
#pragma unroll
    for (int r = 0; r < 15; ++r) {
        const T t = ((valid >> r) & 1u) ? load(r) : T(0);
        if constexpr (sizeof(T) == 4) k[r] = __float_as_int(t);
        else k[r] = __double_as_longlong(t);
        signs |= k[r];
    }
    if (signs < 0) {
#pragma unroll
        for (int r = 0; r < 15; ++r) {
            const K m = k[r] >> (8 * sizeof(K) - 1);
            k[r] = ((k[r] & kHigh) ^ m) - m;
        }
    }
    asc = desc = kSelf;
    K hi = kLow, lo = kHigh;  // (beyond the keys of all values)
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int r = 0; r < 15; ++r) {
            const bool in = ((valid >> r) & 1u) != 0u;
            hi = max(hi, in ? k[r] : kLow);
            lo = min(lo, in ? k[r] : kHigh);
        }
#pragma unroll
        for (int r = 0; r < 15; ++r) {
            if (((valid >> r) & 1u) && k[r] == hi) asc = r;
            if (((valid >> (14 - r)) & 1u) && k[14 - r] == lo) desc = 14 - r;
        }
    } else {
#pragma unroll
        for (int r = 0; r < 15; ++r) {
            const bool in = ((valid >> r) & 1u) != 0u;
            if (in && k[r] >= hi) { hi = k[r]; asc = r; }
            if (in && k[r] < lo) { lo = k[r]; desc = r; }
        }
    }
}

// The same on the field in global memory.
template <typename T, bool NANS>
__device__ __forceinline__ void exact_ranks(const T *__restrict__ v, size_t i, const Geom &g, uint32_t valid,
                                            int &asc, int &desc) {
    const ptrdiff_t sy = g.nx, sz = static_cast<ptrdiff_t>(g.nx) * g.ny;
    const T *c = v + i;
    scan_ranks<T, NANS, 5>([&](int r) { return __ldg(c + (rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz)); }, valid, asc, desc);
}

// What a march reads and writes.  kFirst: f and fhat in, codes, the proxies
// hp (fp64), requests and mismatch bits out.  kDetect: fhat and the codes in,
// requests out, of every voxel.  kCodes: f in, codes out.  kPair: f and fh in, both
// codes out and their differences counted, the values compared with a bound:
// 71.5 M voxels fp64 684 us, where the codes of either field and a pass that
// compares them took 658 + 308.
template <typename T>
struct MarchArgs {
    const T *f, *fh;
    uint8_t *codes;
    uint32_t *hp, *req, *act_next;
    SweepSlot *slot;
    uint8_t *freq = nullptr, *fact = nullptr;  // or null: the group flags of req / act_next
    // kPair: fh's codes; the bound and its magnitude bits (0 unless positive and
    // finite); counters += voxels whose codes differ, of those the ones whose
    // extremum kind does, beyond the bound, beyond the clamp; [4], [5] = 1 if
    // some ascent / descent differs
    uint8_t *codes_h = nullptr;
    T eps = T(0);
    uint64_t sure = 0;
    unsigned long long *pair = nullptr;
};

__device__ __forceinline__ uint64_t bits_mag(double v) {
    return static_cast<uint64_t>(__double_as_longlong(v)) & 0x7FFFFFFFFFFFFFFFull;
}
__device__ __forceinline__ uint64_t bits_mag(float v) { return __float_as_uint(v) & 0x7FFFFFFFu; }

constexpr int kMHY = kMY + 2;        // rows of a tile, and with the halo
constexpr int kMCells = kHX * kMHY;            // cells of a tile's plane
constexpr int kPerThread = (kMCells + kThreads - 1) / kThreads;
// Planes of proxies (k-1, k, then k+1 over k-2): plane k is in slot k mod 3,
// and the plane loop carries the slot along.  Raw stages: the planes k+1 and k+2
// are in flight while plane k is computed, and the passes over one field keep
// the values of k-2, k-1 and k as well, for the decisions in place.
constexpr int kRing = 3;
constexpr int raw_stages(int fields) { return fields == 1 ? 5 : kRing; }
static_assert(kMarchMaxDepth <= 128 && kMY <= 16, "queue entries hold 7 bits of depth and 4 of the row");
constexpr uint32_t kQueueFlush = 256;          // a queue longer than this is emptied after the plane
constexpr uint32_t kQueueCap = kQueueFlush + 2 * kThreads;
// One field: as many failed certificates within this many planes (a quarter of
// their voxels; three quarters of one plane's) take the rest of a column to
// march_tied.  At 255 in four planes, fields of ties take up to 3 % longer, at 128
// in two, fields with some 4 %.
constexpr uint32_t kTiedFlush = 192;
constexpr int kTiedPlanes = 3;
static_assert(kTiedFlush <= kQueueFlush, "the queue holds what is appended before it is emptied");

// Queue entries: tx | row << 5 | (z - zb) << 9 | b << 16 | c << 24 with c the
// code byte of the original.  Rules: b = the current field's tag differences.
// Exact: b = kKnown if c is known, else kUnknown; in the fp64 first pass the current
// field's tag differences (neither is 8) where both certificates hold and a value
// of the stencil is out of the plain range: only this voxel's own are looked at
// then (a 256^3 field of values beyond 1e30: 1840 -> 1585 us).
constexpr uint32_t kKnown = 0x88u, kUnknown = 0x08u;
template <typename T, int MODE>
constexpr bool kOpenRange = MODE == kFirst && sizeof(T) == 8;
template <typename T, int NF>
struct MarchSmem {
    uint32_t p[kRing][NF][kMCells];  // tagged proxies
    uint32_t xq[kQueueCap], rq[kQueueCap];
    uint32_t qn;                           // queue lengths: rules, exact << 16
    uint32_t cnt[3];                       // fmax, fmin, fdir
    uint32_t active, bad;
    uint32_t pair[6];                      // kPair's counters
    // requests of planes zb-1 .. ze, rows y0-1 .. y0+8: a word of the columns
    // x0 .. x0+31, and two bits for the columns x0-1 and x0+32; mismatch bits
    // of the tile's own rows
    uint32_t req[(kMarchMaxDepth + 2) * kMHY], edge[((kMarchMaxDepth + 2) * kMHY + 15) / 16], mism[kMarchMaxDepth * kMY];
    uint8_t lut[256];                      // tag differences of the steepest pair -> code byte
    MarchArgs<T> a;                        // for march_queues
    Geom g;
    int x0, y0, zb;
};
template <typename T, int MODE>
using MarchSmemOf = MarchSmem<T, march_pair(MODE) ? 2 : 1>;

// dx + 1, dy + 1, dz + 1 of every rank, two bits each.
constexpr uint32_t step_bits(int axis) {
    uint32_t t = 0;
    for (int r = 0; r < 15; ++r)
        t |= static_cast<uint32_t>((axis == 0 ? rank_dx(r) : axis == 1 ? rank_dy(r) : rank_dz(r)) + 1) << (2 * r);
    return t;
}
constexpr uint32_t kStepX = step_bits(0), kStepY = step_bits(1), kStepZ = step_bits(2);

// Decides the queued voxels of the block (every thread calls it, behind a
// barrier).  Not inlined: its registers stay out of the plane loop, whose
// state lives across the rare calls from inside it.
template <typename T, int MODE>
__device__ __noinline__ void march_queues(MarchSmemOf<T, MODE> &sm) {
    const int tid = threadIdx.y * kTX + threadIdx.x;
    const MarchArgs<T> &a = sm.a;
    const Geom &g = sm.g;
    const int x0 = sm.x0, y0 = sm.y0, zb = sm.zb;
    uint32_t cmax = 0, cmin = 0, cdir = 0;
    // the voxel (lx, ly, lz) of the tile: requests and mismatch bits go to the
    // column's bitmaps in shared memory
    auto outcome = [&](int lx, int ly, int lz, uint32_t asc, uint32_t desc, uint32_t c) {
        uint32_t tm = detect_rules(static_cast<int>(asc), static_cast<int>(desc), static_cast<int>(c & 15u),
                                   static_cast<int>(c >> 4), cmax, cmin, cdir);
        if (!tm) return;
        if (MODE == kFirst) atomicOr(&sm.mism[lz * kMY + ly], 1u << lx);
        for (; tm; tm &= tm - 1) {
            const uint32_t r2 = 2u * static_cast<uint32_t>(__ffs(tm) - 1);
            const int cx = lx + static_cast<int>((kStepX >> r2) & 3u) - 1;
            const uint32_t cell = static_cast<uint32_t>((lz + static_cast<int>((kStepZ >> r2) & 3u)) * kMHY + ly) +
                                  ((kStepY >> r2) & 3u);
            if (static_cast<unsigned>(cx) < 32u) atomicOr(&sm.req[cell], 1u << cx);
            else atomicOr(&sm.edge[cell >> 4], (cx < 0 ? 1u : 2u) << (2u * (cell & 15u)));
        }
    };
    // kPair: the codes of one voxel in both fields (cmax: they differ; cmin: as
    // extrema; cdir: some ascent, some descent)
    auto differ = [&](uint32_t c0, uint32_t c1) {
        cmax += c0 != c1;
        cmin += ((c0 & 15u) == kSelf) != ((c1 & 15u) == kSelf) || ((c0 >> 4) == kSelf) != ((c1 >> 4) == kSelf);
        cdir |= ((c0 ^ c1) & 15u ? 1u : 0u) | ((c0 ^ c1) >> 4 ? 2u : 0u);
    };
    const uint32_t nx = sm.qn >> 16, nr = sm.qn & 0xFFFFu;
    for (uint32_t j = tid; j < nx; j += kThreads) {
        const uint32_t e = sm.xq[j];
        const int x = x0 + static_cast<int>(e & 31u), y = y0 + static_cast<int>((e >> 5) & 15u),
                  z = zb + static_cast<int>((e >> 9) & 127u);
        const size_t i = flat(g, x, y, z);
        const uint32_t valid = valid_mask(x, y, z, g.nx, g.ny, g.nz);
        uint32_t c = e >> 24;
        int asc, desc;
        if (MODE == kFirst && (bad_value(__ldg(a.f + i)) || bad_value(__ldg(a.fh + i)))) atomicAdd(&sm.bad, 1u);
        const uint32_t b = (e >> 16) & 0xFFu;
        if (kOpenRange<T, MODE> && (b & 15u) != 8u) {
            const uint32_t now = sm.lut[b];
            outcome(x - x0, y - y0, z - zb, now & 15u, now >> 4, c);
            continue;
        }
        if (!march_edits(MODE) || (MODE == kFirst && b == kUnknown)) {
            exact_ranks<T, !march_edits(MODE)>(a.f, i, g, valid, asc, desc);
            c = static_cast<uint32_t>(asc | (desc << 4));
            a.codes[i] = static_cast<uint8_t>(c);
        }
        if (MODE == kPair) {
            exact_ranks<T, true>(a.fh, i, g, valid, asc, desc);
            const uint32_t ch = static_cast<uint32_t>(asc | (desc << 4));
            a.codes_h[i] = static_cast<uint8_t>(ch);
            differ(c, ch);
        }
        if (march_edits(MODE)) {
            exact_ranks<T, false>(a.fh, i, g, valid, asc, desc);
            outcome(x - x0, y - y0, z - zb, static_cast<uint32_t>(asc), static_cast<uint32_t>(desc), c);
        }
    }
    for (uint32_t j = tid; MODE != kCodes && j < nr; j += kThreads) {
        const uint32_t e = sm.rq[j];
        const uint32_t now = sm.lut[(e >> 16) & 0xFFu];
        if (MODE == kPair) {
            differ(e >> 24, now);
            continue;
        }
        outcome(static_cast<int>(e & 31u), static_cast<int>((e >> 5) & 15u), static_cast<int>((e >> 9) & 127u), now & 15u,
                now >> 4, e >> 24);
    }
    if (MODE == kCodes) return;
    if (MODE == kPair) {
        if (cmax) atomicAdd(&sm.pair[0], cmax);
        if (cmin) atomicAdd(&sm.pair[1], cmin);
        if (cdir & 1u) sm.pair[4] = 1;
        if (cdir & 2u) sm.pair[5] = 1;
        return;
    }
    const uint32_t v[3] = {cmax, cmin, cdir};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint32_t t = warp_sum_u32(v[c]);
        if (threadIdx.x == 0 && t) atomicAdd(&sm.cnt[c], t);
    }
}

// Proxies outside [lo, hi) may belong to a NaN or to the sentinel 1e30 (fp64).
// A NaN of high word 0xFFF00000 has the proxy of -inf, which is thus outside.
template <typename T> struct PlainRange;
template <> struct PlainRange<double> {
    static constexpr uint32_t lo = 0x00100010u, hi = (0x80000000u + 0x46293E59u) & ~15u;  // 1e30 = 0x46293E59...
};
template <> struct PlainRange<float> {
    static constexpr uint32_t lo = 0x00800000u, hi = 0xFF800000u;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The rest of a column of one field, from plane k on (the voxels of plane k-1), where
// many certificates fail, as on plateaus: every voxel is decided on the values
// of the raw stages, with no proxies, and no queue but for the rules.  Through
// the queue such a voxel costs about as much as six certified ones: its gather from
// global memory, and the state rebuilt each time the queue is emptied.
// Direction codes, queue -> here: 32 M voxels quantised to a hundred values fp32
// 724 -> 312 us, fp64 1046 -> 478 (unquantised 165 and 174); a ramp of 17 M, all
// ties, 386 -> 222 and 580 -> 291.  Four detections of 256^3 fp64 plateaus, every
// voxel asking for edits: 2.9 -> 2.2 ms with their edits.  Bound by the ALU pipe:
// about 80 (fp32) or 160 (fp64) compares and selects per voxel on half-rate units;
// decided row by row inside the certified loop, both rows at once or out of
// line, that loop or this one took 5 to 20 % longer.
template <typename T, int MODE, bool FACE, class SRC>
__device__ __forceinline__ void march_tied(MarchSmemOf<T, MODE> &sm, SRC &src, const MarchArgs<T> &a, const Geom &g, int x,
                                           int y, int zb, int ctr, bool vin0, bool vin1, int k, int nplanes, int stage,
                                           size_t i) {
    constexpr int kStages = raw_stages(1);
    const int tx = threadIdx.x, ty = threadIdx.y;
    const size_t plane = static_cast<size_t>(g.nx) * g.ny;
    auto stage_of = [&](int ahead) { return stage + ahead < kStages ? stage + ahead : stage + ahead - kStages; };
#pragma unroll 1
    while (k < nplanes) {
        src.prefetch(k + 2, stage_of(2));
        const int zrel = k - 2;
        const T *z0 = src.values(stage_of(3)) + ctr, *z1 = src.values(stage_of(4)) + ctr, *z2 = src.values(stage) + ctr;
        bool over = false;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool vin = r ? vin1 : vin0;
            const size_t ir = i + (r ? static_cast<size_t>(g.nx) : 0);
            uint32_t c = 0, code = 0;
            if (vin) {
                if (MODE == kDetect) c = a.codes[ir];
                int asc, desc;
                scan_tile<T>([&](int q) {
                    return (rank_dz(q) < 0 ? z0 : rank_dz(q) > 0 ? z2 : z1)[rank_dx(q) + (rank_dy(q) + r) * kHX];
                }, FACE ? valid_mask(x, y + r, zb + zrel, g.nx, g.ny, g.nz) : kAllValid, asc, desc);
                code = static_cast<uint32_t>(asc | (desc << 4));
                if (MODE == kCodes) a.codes[ir] = static_cast<uint8_t>(code);
            }
            if constexpr (MODE == kDetect) {
                const bool rule = vin && (code != c || (FACE && c == 0x77u));
                const uint32_t wr = __ballot_sync(0xFFFFFFFFu, rule);
                if (wr) {
                    uint32_t base = 0;
                    if (tx == 0) base = atomicAdd(&sm.qn, static_cast<uint32_t>(__popc(wr)));
                    base = __shfl_sync(0xFFFFFFFFu, base, 0);
                    if (rule)
                        sm.rq[base + static_cast<uint32_t>(__popc(wr & ((1u << tx) - 1u)))] =
                            static_cast<uint32_t>(tx) | (static_cast<uint32_t>(2 * ty + r) << 5) |
                            (static_cast<uint32_t>(zrel) << 9) | (rank_pair_tags(code) << 16) | (c << 24);
                    over |= base + static_cast<uint32_t>(__popc(wr)) > kQueueFlush;
                }
            }
        }
        i += plane;
        if (k + 1 < nplanes) src.wait(0, 0u);
        over = __syncthreads_or(over) != 0;
        ++k;
        stage = stage_of(1);
        if (MODE == kDetect && over) {
            march_queues<T, MODE>(sm);
            __syncthreads();
            if (threadIdx.x == 0 && ty == 0) sm.qn = 0;
            __syncthreads();
        }
    }
    if (MODE == kDetect) march_queues<T, MODE>(sm);
}

// FACE: a block on a domain face, or one whose tile crosses the domain's far
// end; the other blocks' tile, halo and planes zb-1 .. ze lie inside.
template <typename T, int MODE, bool FACE, class SRC>
__device__ __forceinline__ void march_body(MarchSmemOf<T, MODE> &sm, SRC &src, const MarchArgs<T> &a,
                                           const Geom &g, int bx, int by, int bz) {
    constexpr int NF = march_pair(MODE) ? 2 : 1, kStages = raw_stages(NF);
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTX + tx;
    const int x0 = bx * kTX, y0 = by * kMY, zb = bz * g.zc;
    const int ze = FACE ? min(g.nz, zb + g.zc) : zb + g.zc;
    const int x = x0 + tx, y = y0 + 2 * ty;
    const bool vin0 = !FACE || (x < g.nx && y < g.ny), vin1 = !FACE || (x < g.nx && y + 1 < g.ny);
    const size_t plane = static_cast<size_t>(g.nx) * g.ny;
    const int nplanes = ze - zb + 2;  // zb-1 .. ze

    // tags of this thread's cells (tid + 128 j of the 34 x 10 halo tile) in
    // plane zb-1, 4 bits each
    uint32_t ctags = 0;
    uint32_t mine = 0, beyond = 0, clamped = 0;  // kPair: cells of the tile itself; values beyond the bound, the clamp
#pragma unroll
    for (int j = 0; j < kPerThread; ++j) {
        const int c = tid + j * kThreads;
        const int cy = c / kHX, cx = c - cy * kHX;
        ctags |= stencil_tag(x0 - 1 + cx, y0 - 1 + cy, zb - 1) << (8 * j);
        if (MODE == kPair && c < kMCells && cx >= 1 && cx <= kTX && cy >= 1 && cy <= kMY && x0 - 1 + cx < g.nx &&
            y0 - 1 + cy < g.ny)
            mine |= 1u << j;
    }
    auto plane_in = [&](int k) { return !FACE || (zb - 1 + k >= 0 && zb - 1 + k < g.nz); };
    auto convert = [&](int k, int slot, int stage, uint32_t parity) {
        src.wait(stage, parity);
        if (!plane_in(k)) return;
        uint32_t *dst = &sm.p[slot][0][tid];
        const uint32_t tags = ctags + 0x020202u * (static_cast<uint32_t>(k) & 7u);
#pragma unroll
        for (int j = 0; j < kPerThread; ++j) {
            if (j == kPerThread - 1 && tid + j * kThreads >= kMCells) break;
            const uint32_t tag = (tags >> (8 * j)) & 15u;
#pragma unroll
            for (int F = 0; F < NF; ++F) dst[F * kMCells + j * kThreads] = proxy_of(src.cell(stage, j, F)) | tag;
            if constexpr (MODE == kPair) {
                // One subtraction decides nearly all (GB300's fp64 pipe runs two
                // operations per SM and cycle): fl(p - f) rounds monotonically
                // and eps is representable, so |fl(p - f)| < eps means
                // |p - f| < eps, and then p lies within [fl(f - eps), fl(f + eps)].
                if (((mine >> j) & 1u) && k >= 1 && k < nplanes - 1) {
                    const T fv = src.cell(stage, j, 0), pv = src.cell(stage, j, 1), d = pv - fv;
                    if (bits_mag(d) >= a.sure) {  // NaN included
                        beyond += !(fabs(d) <= a.eps);
                        clamped += !(pv >= fv - a.eps && pv <= fv + a.eps);
                    }
                }
            }
        }
    };
    // The cells a plane contributes, from the centre cell of the lower voxel.
    // On a face the step outside the domain is left out, which reads another
    // cell of the same block a second time.
    const int ctr = (2 * ty + 1) * kHX + tx + 1;
    const int xm = FACE && x == 0 ? 0 : -1, xp = FACE && x + 1 >= g.nx ? 0 : 1;
    const int ra = FACE && y == 0 ? 0 : -kHX, rc = FACE && y + 1 >= g.ny ? 0 : kHX,
              rd = FACE && y + 2 >= g.ny ? rc : 2 * kHX;
    // the blocks U and V of the two voxels in a plane, on the values with
    // their tags flipped by `flip`
    struct Blocks {
        Ext2 u0, u1, v0, v1;
    };
    auto blocks = [&](const uint32_t *t, uint32_t flip) {
        const uint32_t a0 = t[ra] ^ flip, a1 = t[ra + xp] ^ flip;
        const uint32_t bm = t[xm] ^ flip, b0 = t[0] ^ flip, b1 = t[xp] ^ flip;
        const uint32_t cm = t[rc + xm] ^ flip, c0 = t[rc] ^ flip, c1 = t[rc + xp] ^ flip;
        const uint32_t dm = t[rd + xm] ^ flip, d0 = t[rd] ^ flip;
        const Ext2 p1 = ext2(b0, b1), q1 = ext2(cm, c0);
        return Blocks{join(a0, a1, p1), join(c0, c1, p1), join(bm, b0, q1), join(dm, d0, q1)};
    };

    if (tid == 0) {
        sm.qn = 0;
        sm.cnt[0] = sm.cnt[1] = sm.cnt[2] = 0;
        sm.active = sm.bad = 0;
        if (MODE == kPair)
            for (int c = 0; c < 6; ++c) sm.pair[c] = 0;
        sm.a = a;
        sm.g = g;
        sm.x0 = x0;
        sm.y0 = y0;
        sm.zb = zb;
    }
    for (int e = tid; e < 256; e += kThreads) sm.lut[e] = tag_pair_code(static_cast<uint32_t>(e));
    if (march_edits(MODE)) {
        for (int e = tid; e < nplanes * kMHY; e += kThreads) sm.req[e] = 0;
        for (int e = tid; e < (nplanes * kMHY + 15) / 16; e += kThreads) sm.edge[e] = 0;
        if (MODE == kFirst)
            for (int e = tid; e < (nplanes - 2) * kMY; e += kThreads) sm.mism[e] = 0;
    }
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {  // at least 3 planes
        convert(k, k, k, 0u);
        if (k == 0) src.prefetch(kRing, kRing % kStages);
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < 3; ++k) src.release(k, k);
    size_t i = static_cast<size_t>(x) + static_cast<size_t>(y) * g.nx + static_cast<size_t>(zb) * plane;
    const uint32_t stag0 = stencil_tag(x, y, zb - 2);
    int k = 2;  // the next plane; it completes the voxels of plane k-1, z = zb + k - 2
    int slot = 2, next = 0;  // of planes k and k+1
    int stage = 2;           // one field: of plane k (two fields: the slots)
    int flushed = 2;         // the plane before which the queues were last empty
    auto stage_of = [&](int ahead) { return stage + ahead < kStages ? stage + ahead : stage + ahead - kStages; };
    uint32_t parity = 1u;    // of plane k+1's stage
#pragma unroll 1
    while (true) {
        // the state before plane k, from the planes still in the ring (also
        // after the queues were emptied, so that nothing lives across that
        // call): [field][tags plain / flipped][voxel]
        Ext2 G[NF][2][2], U[NF][2][2];
#pragma unroll
        for (int F = 0; F < NF; ++F)
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const Blocks w = blocks(&sm.p[3 - slot - next][F][ctr], p ? 15u : 0u);
                U[F][p][0] = w.u0;
                U[F][p][1] = w.u1;
                G[F][p][0] = join(w.u0, w.v0);
                G[F][p][1] = join(w.u1, w.v1);
                if (plane_in(k - 2)) {
                    const Blocks o = blocks(&sm.p[next][F][ctr], p ? 15u : 0u);
                    G[F][p][0] = join(G[F][p][0], o.u0);
                    G[F][p][1] = join(G[F][p][1], o.u1);
                }
            }
        __syncthreads();  // plane k+1 takes the slot of plane k-2, which every thread has read
        bool over = false;
#pragma unroll 1
        while (!over && k < nplanes) {
            const int last = 3 - slot - next;  // the slot of plane k-1, and of k+2's stage
            src.prefetch(k + 2, NF == 1 ? stage_of(2) : last);
            const int zrel = k - 2;
            uint32_t was[2] = {0u, 0u};
            if (MODE == kDetect) {
                if (vin0) was[0] = a.codes[i];
                if (vin1) was[1] = a.codes[i + g.nx];
            }
            Ext2 S[NF][2][2];
            if (plane_in(k)) {
#pragma unroll
                for (int F = 0; F < NF; ++F) {
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const Blocks w = blocks(&sm.p[slot][F][ctr], p ? 15u : 0u);
                        S[F][p][0] = join(G[F][p][0], w.v0);
                        S[F][p][1] = join(G[F][p][1], w.v1);
                        G[F][p][0] = join(U[F][p][0], w.u0, w.v0);
                        G[F][p][1] = join(U[F][p][1], w.u1, w.v1);
                        U[F][p][0] = w.u0;
                        U[F][p][1] = w.u1;
                    }
                }
            } else {  // the plane beyond the domain, the last one
#pragma unroll
                for (int F = 0; F < NF; ++F)
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        S[F][p][0] = G[F][p][0];
                        S[F][p][1] = G[F][p][1];
                    }
            }
            const uint32_t stag = stag0 + 2u * static_cast<uint32_t>(k);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const bool vin = r ? vin1 : vin0;
                const size_t ir = i + (r ? static_cast<size_t>(g.nx) : 0);
                if (MODE == kFirst && sizeof(T) == 8 && vin)  // fhat's proxies
                    a.hp[ir] = sm.p[last][NF - 1][ctr + (r ? (FACE ? rc : kHX) : 0)] & ~15u;
                const uint32_t cert0 = (S[0][0][r].hi ^ S[0][1][r].hi) & (S[0][0][r].lo ^ S[0][1][r].lo);
                uint32_t cert = cert0;
                if (NF == 2)
                    cert &= (S[NF - 1][0][r].hi ^ S[NF - 1][1][r].hi) & (S[NF - 1][0][r].lo ^ S[NF - 1][1][r].lo);
                const bool ok0 = (cert0 & 15u) == 15u;
                bool ok = (cert & 15u) == 15u;
                if (MODE == kFirst)
                    ok = ok && max(S[0][0][r].hi, S[NF - 1][0][r].hi) < PlainRange<T>::hi &&
                         min(S[0][0][r].lo, S[NF - 1][0][r].lo) >= PlainRange<T>::lo;
                const uint32_t st = stag + static_cast<uint32_t>(r);
                const uint32_t c0 = sm.lut[((S[0][0][r].hi - st) & 15u) | (((S[0][0][r].lo - st) & 15u) << 4)];
                bool rule = false, ex = vin && !ok;
                uint32_t c = c0;
                if (MODE == kCodes) {
                    if (vin && ok) a.codes[ir] = static_cast<uint8_t>(c0);
                } else if (MODE == kPair) {
                    const uint32_t now = ((S[NF - 1][0][r].hi - st) & 15u) | (((S[NF - 1][0][r].lo - st) & 15u) << 4);
                    if (vin && ok) {
                        a.codes[ir] = static_cast<uint8_t>(c0);
                        a.codes_h[ir] = sm.lut[now];
                    }
                    rule = vin && ok &&
                           (((S[0][0][r].hi ^ S[NF - 1][0][r].hi) | (S[0][0][r].lo ^ S[NF - 1][0][r].lo)) & 15u) != 0u;
                } else if (MODE == kFirst) {
                    if (vin && ok0) a.codes[ir] = static_cast<uint8_t>(c0);
                    // equal codes fire no rule unless the voxel is both maximum
                    // and minimum of f, which a certified voxel is only without
                    // neighbours (a field of one voxel)
                    rule = vin && ok &&
                           ((((S[0][0][r].hi ^ S[NF - 1][0][r].hi) | (S[0][0][r].lo ^ S[NF - 1][0][r].lo)) & 15u) != 0u ||
                            (FACE && c0 == 0x77u));
                } else {
                    c = was[r];
                    rule = vin && ok && (c0 != c || (FACE && c == 0x77u));
                }
                const uint32_t wq = __ballot_sync(0xFFFFFFFFu, rule || ex);
                if (wq) {
                    const uint32_t wx = __ballot_sync(0xFFFFFFFFu, ex), wr = wq & ~wx;
                    const uint32_t lower = (1u << tx) - 1u;
                    uint32_t base = 0;
                    const uint32_t add = static_cast<uint32_t>(__popc(wr)) | (static_cast<uint32_t>(__popc(wx)) << 16);
                    if (tx == 0) base = atomicAdd(&sm.qn, add);
                    base = __shfl_sync(0xFFFFFFFFu, base, 0);
                    const uint32_t here = static_cast<uint32_t>(tx) | (static_cast<uint32_t>(2 * ty + r) << 5) |
                                          (static_cast<uint32_t>(zrel) << 9) | (c << 24);
                    const uint32_t now = ((S[NF - 1][0][r].hi - st) & 15u) | (((S[NF - 1][0][r].lo - st) & 15u) << 4);
                    if (ex) {
                        sm.xq[(base >> 16) + static_cast<uint32_t>(__popc(wx & lower))] =
                            here | ((kOpenRange<T, MODE> && (cert & 15u) == 15u ? now : ok0 ? kKnown : kUnknown) << 16);
                    } else if (rule) {
                        sm.rq[(base & 0xFFFFu) + static_cast<uint32_t>(__popc(wr & lower))] = here | (now << 16);
                    }
                    const uint32_t end = base + add;
                    over |= (end & 0xFFFFu) > kQueueFlush || (end >> 16) > (NF == 1 ? kTiedFlush : kQueueFlush);
                }
            }
            i += plane;
            if (k + 1 < nplanes) convert(k + 1, next, NF == 1 ? stage_of(1) : next, parity);
            // the barrier that ends the plane also tells whether a queue could
            // overflow in the next one (every appending warp knows its end)
            over = __syncthreads_or(over) != 0;
            src.release(k + 1, next);
            ++k;
            if (NF == 1) stage = stage_of(1);
            slot = next;
            next = next == kRing - 1 ? 0 : next + 1;
            if (next == 0) parity ^= 1u;
        }
        const uint32_t queued = sm.qn >> 16;
        march_queues<T, MODE>(sm);
        if (k >= nplanes) break;
        __syncthreads();
        if (tid == 0) sm.qn = 0;
        __syncthreads();
        if constexpr (NF == 1) {
            if (queued > kTiedFlush && k - flushed <= kTiedPlanes) {
                march_tied<T, MODE, FACE>(sm, src, a, g, x, y, zb, ctr, vin0, vin1, k, nplanes, stage, i);
                break;
            }
            flushed = k;
        }
    }
    if (MODE == kCodes) return;
    if (MODE == kPair) {
        beyond = warp_sum_u32(beyond);
        clamped = warp_sum_u32(clamped);
        if (tx == 0 && beyond) atomicAdd(&sm.pair[2], beyond);
        if (tx == 0 && clamped) atomicAdd(&sm.pair[3], clamped);
        __syncthreads();
        if (tid < 4 && sm.pair[tid]) atomicAdd(a.pair + tid, static_cast<unsigned long long>(sm.pair[tid]));
        if ((tid == 4 || tid == 5) && sm.pair[tid]) a.pair[tid] = 1;
        return;
    }
    __syncthreads();
    // the column's bitmaps: one global atomic per word with a request (the
    // neighbouring columns request voxels of this one, too), a plain store per
    // word with a mismatch (its rows are this block's alone)
    for (int e = tid; e < nplanes * kMHY; e += kThreads) {
        const uint32_t m = sm.req[e], ed = (sm.edge[e >> 4] >> (2 * (e & 15))) & 3u;
        if (m | ed) {
            const int pl = e / kMHY, row = e - pl * kMHY;
            const size_t w = word_of(g, x0, y0 - 1 + row, zb - 1 + pl);
            if (m) atomicOr(a.req + w, m);
            if (ed & 1u) atomicOr(a.req + w - 1, 1u << 31);
            if (ed & 2u) atomicOr(a.req + w + 1, 1u);
            if (a.freq) {
                if (m) a.freq[w / kGroupWords] = 1;
                if (ed & 1u) a.freq[(w - 1) / kGroupWords] = 1;
                if (ed & 2u) a.freq[(w + 1) / kGroupWords] = 1;
            }
        }
    }
    for (int e = tid; MODE == kFirst && e < (nplanes - 2) * kMY; e += kThreads)
        if (sm.mism[e]) {
            const size_t w = word_of(g, x0, y0 + e % kMY, zb + e / kMY);
            a.act_next[w] = sm.mism[e];
            if (a.fact) a.fact[w / kGroupWords] = 1;
        }
    const uint32_t active = warp_sum_u32(static_cast<uint32_t>(ze - zb) * ((vin0 ? 1u : 0u) + (vin1 ? 1u : 0u)));
    if (tx == 0 && active) atomicAdd(&sm.active, active);
    __syncthreads();
    // one atomic per non-zero counter and block
    if (tid < 3 && sm.cnt[tid]) atomicAdd(reinterpret_cast<unsigned long long *>(a.slot) + tid, static_cast<unsigned long long>(sm.cnt[tid]));
    if (tid == 3 && sm.active) atomicAdd(&a.slot->active, static_cast<unsigned long long>(sm.active));
    if (tid == 4 && sm.bad) atomicAdd(&a.slot->bad, static_cast<unsigned long long>(sm.bad));
}

__device__ __forceinline__ bool march_inside(const Geom &g, int bx, int by, int bz) {
    const int x0 = bx * kTX, y0 = by * kMY, zb = bz * g.zc;
    return x0 >= 1 && x0 + kTX + 1 <= g.nx && y0 >= 1 && y0 + kMY + 1 <= g.ny && zb >= 1 && zb + g.zc + 1 <= g.nz;
}

// ---------------------------------------------------------------------------
// Plane sources.  cell(k, j, F): this thread's cell tid + 128 j of the halo
// tile, of field F, in plane zb-1+k.
//
// CopySource: cp.async of single elements, any alignment and row length; every
// thread copies and later converts its own cells, so a plane needs no barrier
// between its arrival and its conversion.  prefetch(k) starts plane k into a
// stage whose plane this thread has converted and, of one field, no thread reads
// any more.  values(s): the tile in stage s, cell after cell.
// ---------------------------------------------------------------------------
template <typename R, int NF>
struct CopyTile {
    R raw[raw_stages(NF)][NF][kMCells];
};

template <typename R, int NF, bool FACE>
struct CopySource {
    CopyTile<R, NF> *ct;
    const R *v0, *v1;
    size_t plane;
    size_t off[kPerThread];  // of this thread's cells in their plane
    uint32_t in;             // bit j: cell j lies inside the domain
    int zb, nz, nplanes;
    __device__ __forceinline__ CopySource(CopyTile<R, NF> &t, const R *f0, const R *f1, const Geom &g, int bx, int by,
                                          int bz)
        : ct(&t), v0(f0), v1(f1), plane(static_cast<size_t>(g.nx) * g.ny), in(0), zb(bz * g.zc), nz(g.nz),
          nplanes((FACE ? min(g.nz, bz * g.zc + g.zc) - bz * g.zc : g.zc) + 2) {
        const int tid = threadIdx.y * kTX + threadIdx.x;
#pragma unroll
        for (int j = 0; j < kPerThread; ++j) {
            const int c = tid + j * kThreads;
            const int cy = c / kHX, cx = c - cy * kHX;
            const int gx = bx * kTX - 1 + cx, gy = by * kMY - 1 + cy;
            const bool ok = c < kMCells && (!FACE || (gx >= 0 && gx < g.nx && gy >= 0 && gy < g.ny));
            if (ok) in |= 1u << j;
            off[j] = ok ? static_cast<size_t>(gx) + static_cast<size_t>(gy) * g.nx : 0;
        }
#pragma unroll 1
        for (int k = 0; k < kRing; ++k) prefetch(k, k);
    }
    __device__ __forceinline__ void prefetch(int k, int s) {
        if (k < nplanes && (!FACE || (zb - 1 + k >= 0 && zb - 1 + k < nz))) {
            const size_t zo = static_cast<size_t>(zb - 1 + k) * plane;
            const int tid = threadIdx.y * kTX + threadIdx.x;
#pragma unroll
            for (int j = 0; j < kPerThread; ++j)
                if ((in >> j) & 1u)
#pragma unroll
                    for (int F = 0; F < NF; ++F)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                                         smem_u32(&ct->raw[s][F][tid + j * kThreads])),
                                     "l"((F == 0 ? v0 : v1) + zo + off[j]), "n"(static_cast<int>(sizeof(R)))
                                     : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");  // one group per plane, also when empty
    }
    // plane k has arrived: when it is converted, planes up to k + 1 have been started
    __device__ __forceinline__ void wait(int, uint32_t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
    }
    __device__ __forceinline__ R cell(int s, int j, int F) const {
        return ct->raw[s][F][threadIdx.y * kTX + threadIdx.x + j * kThreads];
    }
    __device__ __forceinline__ const R *values(int s) const { return ct->raw[s][0]; }
    __device__ __forceinline__ void release(int, int) {}
};

template <typename T, int MODE>
struct CopyMarch {  // shared memory of a copy-fed march
    CopyTile<T, march_pair(MODE) ? 2 : 1> raw;
    MarchSmemOf<T, MODE> m;
};

template <typename T, int MODE, bool FACE>
__device__ __forceinline__ void march_copies(CopyMarch<T, MODE> &sm, const MarchArgs<T> &a, const Geom &g, int bx,
                                             int by, int bz) {
    CopySource<T, march_pair(MODE) ? 2 : 1, FACE> s(sm.raw, MODE == kDetect ? a.fh : a.f, a.fh, g, bx, by, bz);
    march_body<T, MODE, FACE>(sm.m, s, a, g, bx, by, bz);
}

// bz0: index of the first z-chunk the launch covers (a launch may cover a
// z-range of chunks, e.g. the part of the field already copied in).
// Six blocks per SM with one field (codes 512^3 fp64 611 -> 587 us, fp32 564 -> 552),
// five with two, whose state does not fit 80 registers.
template <typename T, int MODE>
__global__ void __launch_bounds__(kThreads, march_pair(MODE) ? 5 : 6) k_march(const __grid_constant__ MarchArgs<T> a,
                                                       const __grid_constant__ Geom g, int bz0) {
    extern __shared__ __align__(128) unsigned char march_smem[];
    CopyMarch<T, MODE> &sm = *reinterpret_cast<CopyMarch<T, MODE> *>(march_smem);
    const int bx = static_cast<int>(blockIdx.x), by = static_cast<int>(blockIdx.y),
              bz = bz0 + static_cast<int>(blockIdx.z);
    if (march_inside(g, bx, by, bz))
        march_copies<T, MODE, false>(sm, a, g, bx, by, bz);
    else
        march_copies<T, MODE, true>(sm, a, g, bx, by, bz);
}

// ---------------------------------------------------------------------------
// Thin fields, kCodes and kDetect: one voxel per thread in storage order, its 15
// values gathered.  A march works on 32 x 8 planes whatever part of them the field
// fills, and of a field of one plane on three: a line of 2 M voxels is 62 500
// blocks of 32 voxels.  The gathers win below a third of the cells in use (codes
// of 2 M fp32 voxels, march and here: 1/8, a line, 180 and 38 us; 1/4, four planes two
// voxels high, 65 and 44; 3/8, 300 planes three high, 53 and 45, but fp64 55 and
// 60), in a single plane up to a half (four rows: 64 and 42, fp64 68 and 49; eight:
// 45 and 41, 47 and 51).
// ---------------------------------------------------------------------------
inline bool march_thin(const Geom &g) {
    const uint64_t used = static_cast<uint64_t>(g.nx) * static_cast<uint64_t>(g.ny),
                   cells = column_planes(static_cast<size_t>(g.nx), static_cast<size_t>(g.ny), 1) * kTX * kMY;
    return g.n < (static_cast<size_t>(1) << 32) && (3 * used < cells || (g.nz == 1 && 2 * used <= cells));
}

template <typename T, int MODE>
__global__ void __launch_bounds__(256) k_flat(const __grid_constant__ MarchArgs<T> a, const __grid_constant__ Geom g) {
    uint32_t cmax = 0, cmin = 0, cdir = 0, active = 0;
    const uint32_t n = static_cast<uint32_t>(g.n), step = gridDim.x * 256u;
    for (uint64_t at = blockIdx.x * 256u + threadIdx.x; at < n; at += step) {
        const uint32_t i = static_cast<uint32_t>(at), row = fdiv(i, g.div_nx), zz = fdiv(row, g.div_ny);
        const int x = static_cast<int>(i - row * static_cast<uint32_t>(g.nx)),
                  y = static_cast<int>(row - zz * static_cast<uint32_t>(g.ny)), z = static_cast<int>(zz);
        int asc, desc;
        exact_ranks<T, MODE == kCodes>(MODE == kCodes ? a.f : a.fh, i, g, valid_mask(x, y, z, g.nx, g.ny, g.nz), asc, desc);
        if (MODE == kCodes) {
            a.codes[i] = static_cast<uint8_t>(asc | (desc << 4));
        } else {
            const uint8_t c = a.codes[i];
            request_targets(a.req, g, x, y, z, detect_rules(asc, desc, c & 15, c >> 4, cmax, cmin, cdir));
            ++active;
        }
    }
    if (MODE == kDetect) {
        const uint32_t v[8] = {cmax, cmin, cdir, 0u, 0u, 0u, active, 0u};
        block_flush_slot(a.slot, v);
    }
}

// ---------------------------------------------------------------------------
// TmaSource (two fields): one thread issues, per plane, a
// cp.async.bulk.tensor box of f and one of fhat (the tile with its one-voxel
// halo, widened in x so that the box starts on a 16-byte boundary) into the
// stage, guarded by an mbarrier that the copy engine completes with the box's
// byte count; a stage is refilled with the plane three ahead after the
// barrier that ends its conversion.  No thread computes a global address or
// predicates a load for the tile.  Planes outside the domain are not copied:
// their stage's barrier gets a plain arrive.
//
// Every mbarrier wait is bounded: a plane that does not arrive within the
// limit sets *err (the host reports PMSZ_ERR_CUDA), and the block still waits,
// again bounded, on every plane it issued before it exits.
// ---------------------------------------------------------------------------
template <typename T> struct RawBox;
template <> struct RawBox<double> { static constexpr int kX = 36, kOff = 1; };  // x0-2 .. x0+33
template <> struct RawBox<float> { static constexpr int kX = 40, kOff = 3; };   // x0-4 .. x0+35
template <typename T>
constexpr int kRawBytes = RawBox<T>::kX * kMHY * static_cast<int>(sizeof(T));  // one box of one field
template <typename T>
constexpr int kRawPitch = (kRawBytes<T> + 127) / 128 * 128;  // stages start on 128-byte boundaries

template <typename T>
struct __align__(128) TmaMarch {
    // first: the copy engine writes the stages, which must start on 128-byte
    // boundaries (the struct is 128-byte aligned, kRawPitch a multiple of 128)
    alignas(128) unsigned char raw[kRing][2][kRawPitch<T>];  // boxes of f and fhat, rows of RawBox<T>::kX
    MarchSmem<T, 2> m;
    unsigned long long mbar[kRing];
};
static_assert(offsetof(TmaMarch<float>, raw) == 0 && offsetof(TmaMarch<double>, raw) == 0 &&
                  kRawPitch<float> % 128 == 0 && kRawPitch<double> % 128 == 0,
              "TMA stages must start on 128-byte boundaries");

constexpr int kMbarTries = 1 << 22;  // try_wait suspends between tries: a bound of seconds, not a spin count

__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity) {
    for (int it = 0; it < kMbarTries; ++it) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t mbar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 :: "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(mbar) : "memory");
}

template <typename T, bool FACE>
struct TmaSource {
    TmaMarch<T> *sm;
    const CUtensorMap *tf, *tfh;
    int x0, y0, zb, nz, nplanes;
    int r[kPerThread];  // this thread's cells in a box
    uint32_t failed;
    __device__ __forceinline__ void issue(int k, int s) {  // plane zb-1+k into stage s = k mod 3 (one thread)
        const uint32_t mb = smem_u32(&sm->mbar[s]);
        if (FACE && (zb - 1 + k < 0 || zb - 1 + k >= nz)) {  // nothing to copy: complete the phase
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(mb) : "memory");
            return;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the stage's reads come first
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(mb), "r"(2 * kRawBytes<T>)
                     : "memory");
        tma_load_3d(smem_u32(sm->raw[s][0]), tf, x0 - RawBox<T>::kOff - 1, y0 - 1, zb - 1 + k, mb);
        tma_load_3d(smem_u32(sm->raw[s][1]), tfh, x0 - RawBox<T>::kOff - 1, y0 - 1, zb - 1 + k, mb);
    }
    __device__ __forceinline__ void prefetch(int, int) {}
    __device__ __forceinline__ void wait(int s, uint32_t parity) {
        if (!mbar_wait(smem_u32(&sm->mbar[s]), parity)) failed = 1;
    }
    __device__ __forceinline__ T cell(int s, int j, int F) const {
        return reinterpret_cast<const T *>(sm->raw[s][F])[r[j]];
    }
    __device__ __forceinline__ void release(int k, int s) {  // plane k is converted: its stage takes plane k + 3
        if (threadIdx.x == 0 && threadIdx.y == 0 && k + kRing < nplanes) issue(k + kRing, s);
    }
};

template <typename T, int MODE, bool FACE>
__device__ __forceinline__ void pair_tma_body(TmaMarch<T> &sm, const CUtensorMap *tf, const CUtensorMap *tfh,
                                               const MarchArgs<T> &a, const Geom &g, int bx, int by, int bz,
                                               uint32_t *err) {
    TmaSource<T, FACE> s;
    s.sm = &sm;
    s.tf = tf;
    s.tfh = tfh;
    s.x0 = bx * kTX;
    s.y0 = by * kMY;
    s.zb = bz * g.zc;
    s.nz = g.nz;
    s.nplanes = (FACE ? min(g.nz, s.zb + g.zc) - s.zb : g.zc) + 2;
    s.failed = 0;
    const int tid = threadIdx.y * kTX + threadIdx.x;
#pragma unroll
    for (int j = 0; j < kPerThread; ++j) {
        const int c = min(tid + j * kThreads, kMCells - 1);
        const int cy = c / kHX, cx = c - cy * kHX;
        s.r[j] = cy * RawBox<T>::kX + cx + RawBox<T>::kOff;
    }
    if (tid == 0) {
        for (int k = 0; k < kRing; ++k)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&sm.mbar[k])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0)
        for (int k = 0; k < kRing && k < s.nplanes; ++k) s.issue(k, k);
    march_body<T, MODE, FACE>(sm.m, s, a, g, bx, by, bz);
    if (s.failed) atomicOr(err, 1u);
}

// tf / tfh map f / fhat as (nx, ny, nz) with a box of RawBox<T>::kX x kMHY x 1
// (the caller takes k_march where no map can be made: rows whose byte length
// is not a multiple of 16, or base pointers off a 16-byte boundary).
template <typename T, int MODE>  // kFirst or kPair
__global__ void __launch_bounds__(kThreads, 6) k_pair_tma(const __grid_constant__ CUtensorMap tf,
                                                           const __grid_constant__ CUtensorMap tfh,
                                                           const __grid_constant__ MarchArgs<T> a,
                                                           const __grid_constant__ Geom g, int bz0, uint32_t *err) {
    extern __shared__ __align__(128) unsigned char march_smem[];
    TmaMarch<T> &sm = *reinterpret_cast<TmaMarch<T> *>(march_smem);
    const int bx = static_cast<int>(blockIdx.x), by = static_cast<int>(blockIdx.y),
              bz = bz0 + static_cast<int>(blockIdx.z);
    if (march_inside(g, bx, by, bz))
        pair_tma_body<T, MODE, false>(sm, &tf, &tfh, a, g, bx, by, bz, err);
    else
        pair_tma_body<T, MODE, true>(sm, &tf, &tfh, a, g, bx, by, bz, err);
}

inline dim3 tiled_grid(const Geom &g) {
    return dim3(static_cast<unsigned>(g.wpr), static_cast<unsigned>((g.ny + kMY - 1) / kMY),
                static_cast<unsigned>((g.nz + g.zc - 1) / g.zc));
}

// A kernel above the 48 KB of static shared memory has to be allowed its size
// on the current device before it is launched.
template <class K>
inline cudaError_t allow_smem(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(reinterpret_cast<const void *>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(bytes));
}
template <typename T, int MODE>
inline cudaError_t launch_march(dim3 grid, cudaStream_t s, const MarchArgs<T> &a, const Geom &g, int bz0) {
    const cudaError_t e = allow_smem(k_march<T, MODE>, sizeof(CopyMarch<T, MODE>));
    if (e != cudaSuccess) return e;
    k_march<T, MODE><<<grid, dim3(kTX, kThreads / kTX, 1), sizeof(CopyMarch<T, MODE>), s>>>(a, g, bz0);
    return cudaGetLastError();
}

// kCodes or kDetect of a whole field.
template <typename T, int MODE>
inline cudaError_t launch_field(cudaStream_t s, const MarchArgs<T> &a, const Geom &g) {
    if (!march_thin(g)) return launch_march<T, MODE>(tiled_grid(g), s, a, g, 0);
    k_flat<T, MODE><<<static_cast<unsigned>(std::min<size_t>((g.n + 255) / 256, 152 * 16)), 256, 0, s>>>(a, g);
    return cudaGetLastError();
}

}  // namespace pmsz
