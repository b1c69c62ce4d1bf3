// sweep.cuh -- the correction loop's sweeps in one cooperative launch, included
// by correct.cu and sweep_multi.cuh.
//
// The launch takes over behind the fused first pass: the edits of sweep 0, then
// detection and edits sweep after sweep until the stop rule holds, with a grid
// barrier after each phase, every block applying the rule to the same counters.
// No kernel boundary, no compaction into a global list and no host round trip
// between the phases: the bitmaps themselves are the work lists.
//
//  * A flag byte per GROUP of 8 bitmap words (plain stores of 1: no atomics)
//    tells which groups hold anything, so a late sweep reads a byte per 256
//    voxels.
//  * Chunks of groups are dealt round-robin to all threads of the grid,
//    neighbouring chunks to different SMs, so a cluster of activity spreads over
//    the chip.  A block lists its flagged groups in order and its warps take up
//    to four of them at a time as they come free: the wait at the grid barrier
//    was a quarter of the warps' time where each warp kept to its own chunks.
//  * A warp lists the set bits of its four groups in shared memory (each lane
//    the bits of its own word at its prefix) and visits them 32 at a time:
//    nearly full warps whatever the density.
//  * Loads are ordinary cached loads: a grid barrier orders them behind the
//    other blocks' writes, and within a phase no array is both read at
//    neighbours and written (detection reads proxies and codes and writes
//    bitmaps, the edits touch their own voxel's values only), so the 15 gathers
//    of neighbouring voxels share L1 lines.
//  * fp64 detects on the 32-bit proxies; failed certificates wait in a per-warp
//    buffer and are decided on full keys 32 at a time.  fp32 compares the values
//    themselves (the same gathers; 15 values by max and min, then their ranks,
//    cost what the proxies' four chains cost, and nothing is left open), and
//    keeps no proxies: 256^3 dense 3104 -> 2656 us, 120x130x128 983 -> 912, 512^3
//    sparse 2081 -> 1883 against proxies with a switch where many tied.
//  * Result bits collect in shared memory, one word of them per bitmap word
//    (SweepBits), and go out once per four groups: one atomic per word instead
//    of one per voxel, and the closed stencils of all 32 words' changes marked
//    side by side instead of word after word.
//
// Bound by the latency of the gathers (issue slots 40 % used) and, in small
// fields and late sweeps, of the two grid barriers a sweep takes (about 2 us
// each).  Three blocks per SM; fp32 (64 registers) four in large fields, fp64
// with four is up to 8 % slower.  The code is kept small and with one site per
// decision: with dense and sparse visits as two copies the same work took
// 15-25 % longer.
// Whole corrections: list kernels in a conditional CUDA graph -> warps on their
// own chunks, every bit an atomic -> this:
//   64^3 fp32, 8 sweeps              358 -> 181 -> 160 us
//   173x141x203 fp32, 12 sweeps      560 -> 353 -> 282 us
//   512^3 fp64, 16 sparse sweeps    3852 -> 3355 -> 3211 us
//   256^3 fp32, 27 dense sweeps     4727 -> 4467 -> 2656 us
//   160^3 fp64, 40 dense sweeps     2308 -> 2320 -> 1664 us
#pragma once
#include "march.cuh"

namespace pmsz {

constexpr int kSweepBlock = 256, kSweepWarps = kSweepBlock / 32;

__host__ __device__ __forceinline__ size_t group_count(const Geom &g) {
    return (g.nwords + kGroupWords - 1) / kGroupWords;
}

// The stencil's seven rows (dy, dz): (0,0) (1,0) (0,1) (1,1) (-1,0) (0,-1)
// (-1,-1).  Row 0 holds dx = -1, 0, 1; rows 1-3 dx = -1, 0; rows 4-6 dx = 0, 1.
constexpr int kSweepRows = 7;
__host__ __device__ constexpr int step_row(int dy, int dz) {
    return dy == 0 && dz == 0 ? 0 : (dy > 0 || dz > 0 ? 0 : 3) + (dy != 0 ? 1 : 0) + (dz != 0 ? 2 : 0);
}
__device__ __forceinline__ int row_dy(int row) { return row == 1 || row == 3 ? 1 : row == 4 || row == 6 ? -1 : 0; }
__device__ __forceinline__ int row_dz(int row) { return row == 2 || row == 3 ? 1 : row == 5 || row == 6 ? -1 : 0; }
__device__ __forceinline__ uint32_t row_words(const Geom &g, int row) {  // mod 2^32, as word indices are
    return static_cast<uint32_t>(g.wpr) * (static_cast<uint32_t>(row_dy(row)) +
                                           static_cast<uint32_t>(row_dz(row)) * static_cast<uint32_t>(g.ny));
}
// The target of a request by stencil rank (15 entries on 30 banks: no conflicts).
struct SweepStep {
    int dx;       // dx + 1 + 4 * row
    uint32_t dw;  // row_words of the row
};
__device__ __forceinline__ void fill_steps(SweepStep *t, const Geom &g, int lane) {
    if (lane < 15) {
        const uint32_t r2 = 2u * static_cast<uint32_t>(lane);
        const int row = step_row(static_cast<int>((kStepY >> r2) & 3u) - 1, static_cast<int>((kStepZ >> r2) & 3u) - 1);
        t[lane] = {static_cast<int>((kStepX >> r2) & 3u) + 4 * row, row_words(g, row)};
    }
}

// A warp's result bits for the 32 words it visits at a time: the words' own
// (mismatches, changes) and the requests into their seven rows.  Collected
// here they go out as one atomic per word instead of up to three per voxel (L2
// takes one atomic of an address at a time: 160^3 fp64, 40 dense sweeps, 2393 ->
// 2012 us with detection's, -> 1664 us with the edits' and their marks).
struct SweepBits {
    uint32_t own[32], row[kSweepRows][32];  // zero between visits
};

// Marks the closed stencil of the changed bits c of word w (x word wx, row y,
// plane z): the word itself and its six rows' by constant steps from w, the
// neighbouring words only where c reaches them.
__device__ __forceinline__ void mark_words(uint32_t *act, uint8_t *flag, const Geom &g, uint32_t w, int wx, int y, int z,
                                           uint32_t c) {
    const uint32_t tail = wx + 1 == g.wpr ? row_tail_mask(g, wx) : 0xFFFFFFFFu;
    const uint32_t sy = static_cast<uint32_t>(g.wpr), sz = sy * static_cast<uint32_t>(g.ny);
    const bool yp = y + 1 < g.ny, yn = y > 0, zp = z + 1 < g.nz, zn = z > 0;
    auto put = [&](uint32_t at, uint32_t m) {
        atomicOr(act + at, m);
        flag[at / kGroupWords] = 1;
    };
    const uint32_t p = c | (c >> 1), n = (c | (c << 1)) & tail;  // the rows ahead hold dx = -1, 0, the rows behind 0, 1
    put(w, p | n);
    if (yp) put(w + sy, p);
    if (zp) put(w + sz, p);
    if (yp && zp) put(w + sy + sz, p);
    if (yn) put(w - sy, n);
    if (zn) put(w - sz, n);
    if (yn && zn) put(w - sy - sz, n);
    if ((c & 1u) && wx > 0) {
        const uint32_t l = w - 1, m = 1u << 31;
        put(l, m);
        if (yp) put(l + sy, m);
        if (zp) put(l + sz, m);
        if (yp && zp) put(l + sy + sz, m);
    }
    if ((c >> 31) && wx + 1 < g.wpr) {
        const uint32_t r = w + 1;
        put(r, 1u);
        if (yn) put(r - sy, 1u);
        if (zn) put(r - sz, 1u);
        if (yn && zn) put(r - sy - sz, 1u);
    }
}

// State of the sweep loop, ahead of the sweep slots in memory so that one copy
// brings both to the host.
struct LoopState {
    long long k;          // the sweep k_sweeps starts with (the wavefront ran the ones before)
    long long done;       // sweeps in all, once it ends
    int go;               // that sweep runs
    uint32_t err;         // kErrCopy, kErrBarrier
    uint32_t bar[8];      // arrivals at the grid barriers of k_sweeps, and of the wavefront's launches
};
constexpr uint32_t kErrCopy = 1;     // set by the first pass: a tensor copy did not arrive
constexpr uint32_t kErrBarrier = 2;  // set by a sweep kernel: a grid barrier did not complete

// Grid barrier of a cooperative launch: `target` counts the arrivals that
// complete the next one (a counter of the launch's own, zero before it).  The
// arrival returns nothing, so a block polls right behind it; cooperative
// groups' barrier waits for its arrival's answer first (a batch of 32 fields
// 5803 us with that, 5681 with this; a burst of jobs 3998 and 3831).  Bounded:
// all blocks are resident, but if one did not arrive, *err is set and the block
// leaves (the result says so: the caller returns), as every other one then does.
constexpr int kBarrierTries = 1 << 22;  // seconds
__device__ __forceinline__ bool sweep_barrier(uint32_t *bar, uint32_t &target, uint32_t *err) {
    target += gridDim.x;
    __syncthreads();
    int failed = 0;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        int tries = 0;
        uint32_t seen;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
        } while (static_cast<int32_t>(seen - target) < 0 && ++tries < kBarrierTries);
        if (tries == kBarrierTries) {
            atomicOr(err, kErrBarrier);
            failed = 1;
        }
    }
    return __syncthreads_or(failed) == 0;
}

template <typename T>
struct SweepArgs {
    const T *f;
    T *fh;
    const uint8_t *codes;
    uint8_t *cnt;
    uint32_t *hp, *req, *act0, *act1;
    uint8_t *freq, *f0, *f1;  // group flags of req, act0, act1
    SweepSlot *slots;
    LoopState *ls;
    int64_t max_sweeps;
    int from_edits;  // start with the edits of sweep 0 (else with the detection of sweep ls->k, if ls->go)
    Geom g;
    T eps, delta;
    int q;
};

struct SweepSmem {
    uint16_t group[kSweepBlock * 8];      // flagged groups to visit: thread of the chunk * 8 + group in it
    uint32_t groups[kSweepWarps], next;   // listed by each warp, taken
    uint16_t list[kSweepWarps][1024];     // lane of the word << 5 | bit of four groups' set bits
    int4 at[kSweepWarps][32];             // x of bit 0, y, z of their words, and the word
    SweepBits bits[kSweepWarps];
    uint2 defer[kSweepWarps][64];         // word, bit
    SweepStep step[15];
};

// One voxel of a sweep, for A = SweepArgs<T> or Inst<T> (batch.h): the two hold
// a field's pointers and parameters under the same names.
//
// Detection's outcome from the two ranks: detect_rules as two targets, so that
// the lanes of a warp stay together (as a loop over the requested ranks this
// was half of a dense sweep's instructions); the requests and the voxel's
// mismatch bit of the next active set.
template <class A>
__device__ __forceinline__ void sweep_outcome(const A &a, const SweepStep *steps, SweepBits &bits, bool collect, uint32_t *nxt,
                                              uint8_t *fnxt, uint32_t entry, uint32_t w, int asc, int desc, uint8_t c,
                                              uint32_t &cmax, uint32_t &cmin, uint32_t &cdir) {
    if ((asc | (desc << 4)) == static_cast<int>(c) && asc != desc) return;  // (a lone voxel is both: never settled)
    const int oasc = c & 15, odesc = c >> 4;
    const bool omax = oasc == kSelf, omin = !omax && odesc == kSelf;
    const bool r1 = (asc == kSelf) != omax, r2 = (desc == kSelf) != omin, r = r1 || r2;
    const bool v1 = r ? r1 : asc != oasc, v2 = r ? r2 : desc != odesc;
    if (!v1 && !v2) return;
    const uint32_t slot = entry >> 5;
    const int bit = static_cast<int>(entry & 31u);
    cmax += r1;
    cmin += r2;
    cdir += r ? 1u : static_cast<uint32_t>(v1) + static_cast<uint32_t>(v2);
    if (collect) {
        atomicOr(&bits.own[slot], 1u << bit);
    } else {
        atomicOr(nxt + w, 1u << bit);
        fnxt[w / kGroupWords] = 1;
    }
    auto request = [&](int rank) {
        const SweepStep st = steps[rank];
        const int tx = bit + (st.dx & 3) - 1;
        if (collect && static_cast<uint32_t>(tx) < 32u) {
            atomicOr(&bits.row[st.dx >> 2][slot], 1u << tx);
        } else {
            const uint32_t wt = w + st.dw + static_cast<uint32_t>(tx >> 5);
            atomicOr(a.req + wt, 1u << (tx & 31));
            a.freq[wt / kGroupWords] = 1;
        }
    };
    if (v1) request(r1 && !omax ? kSelf : asc);
    if (v2) request(r2 && omin ? kSelf : odesc);
}

// The ranks on full keys (interior: of a warp whose voxels all are; fp32).
template <typename T, class A>
__device__ __forceinline__ void sweep_keys(const A &a, size_t i, int x, int y, int z, bool interior, int &asc, int &desc) {
    const T *c0 = a.fh + i;
    const ptrdiff_t sy = a.g.nx, sz = static_cast<ptrdiff_t>(a.g.nx) * a.g.ny;
    asc = kSelf;
    desc = kSelf;
    if constexpr (sizeof(T) == 4) {
        // The values themselves order fp32 fields (-0 and +0 are equal, a field
        // with NaN ends before its first sweep): the extremes by max and min,
        // NaN standing for a point outside the domain, then the last rank that
        // holds the maximum and the first that holds the minimum.
        T v[15];
        if (interior) {
#pragma unroll
            for (int r = 0; r < 15; ++r) v[r] = c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz];
        } else {
            const uint32_t valid = valid_mask(x, y, z, a.g.nx, a.g.ny, a.g.nz);
#pragma unroll
            for (int r = 0; r < 15; ++r)
                v[r] = ((valid >> r) & 1u) ? c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz] : __int_as_float(0x7FC00000);
        }
        T hi = v[0], lo = v[0];
#pragma unroll
        for (int r = 1; r < 15; r += 2) {
            hi = fmaxf(fmaxf(hi, v[r]), v[r + 1]);
            lo = fminf(fminf(lo, v[r]), v[r + 1]);
        }
#pragma unroll
        for (int r = 0; r < 15; ++r) {
            if (v[r] == hi) asc = r;
            if (v[14 - r] == lo) desc = 14 - r;
        }
        return;
    }
    using K = typename KeyOf<T>::type;
    constexpr int kKeyLoads = 5;  // in flight (fp64 keys are two registers each)
    K hi = 0, lo = ~K(0);
    const uint32_t valid = valid_mask(x, y, z, a.g.nx, a.g.ny, a.g.nz);
#pragma unroll
    for (int r0 = 0; r0 < 15; r0 += kKeyLoads) {
        K kk[kKeyLoads];
#pragma unroll
        for (int j = 0; j < kKeyLoads; ++j) {
            const int r = r0 + j;
            kk[j] = ((valid >> r) & 1u) ? okey(c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz]) : K(0);
        }
#pragma unroll
        for (int j = 0; j < kKeyLoads; ++j)
            if ((valid >> (r0 + j)) & 1u) {
                if (kk[j] >= hi) { hi = kk[j]; asc = r0 + j; }
                if (kk[j] < lo) { lo = kk[j]; desc = r0 + j; }
            }
    }
}
// The ranks on the proxies, with their certificate: of a warp whose voxels are
// all interior (nearly every one: no test per gather), or not.
template <class A>
__device__ __forceinline__ Ext sweep_proxies(const A &a, size_t i) {
    const uint32_t *c0 = a.hp + i;
    const ptrdiff_t sy = a.g.nx, sz = static_cast<ptrdiff_t>(a.g.nx) * a.g.ny;
    uint32_t t[15];
#pragma unroll
    for (int r = 0; r < 15; ++r) t[r] = c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz];
    return proxy_ext_interior(t);
}
template <class A>
__device__ __forceinline__ Ext sweep_proxies_face(const A &a, size_t i, int x, int y, int z) {
    const uint32_t *c0 = a.hp + i;
    const ptrdiff_t sy = a.g.nx, sz = static_cast<ptrdiff_t>(a.g.nx) * a.g.ny;
    uint32_t t[15];
    const uint32_t valid = valid_mask(x, y, z, a.g.nx, a.g.ny, a.g.nz);
#pragma unroll
    for (int r = 0; r < 15; ++r) t[r] = ((valid >> r) & 1u) ? c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz] : 0u;
    return proxy_ext(t);
}
__device__ __forceinline__ bool sweep_interior(const Geom &g, int x, int y, int z) {
    return x >= 1 && x <= g.nx - 2 && y >= 1 && y <= g.ny - 2 && z >= 1 && z <= g.nz - 2;
}
// The edit of one requested voxel (applyDeltaBuffer_local); true if its value changed.
template <typename T, class A>
__device__ __forceinline__ bool sweep_edit(const A &a, size_t v, uint32_t &nreq, uint32_t &nchg, uint32_t &nprog) {
    const T old = a.fh[v];
    const uint8_t oc = a.cnt[v];
    const T fv = __ldg(a.f + v);
    const T lowered = old - a.delta;
    T nv;
    uint8_t nc;
    if (fabs(fv - lowered) <= a.eps && static_cast<int>(oc) < a.q - 1) {
        nv = lowered;
        nc = static_cast<uint8_t>(oc + 1);
    } else {
        nc = static_cast<uint8_t>(a.q);
        nv = fv - a.eps;
    }
    a.fh[v] = nv;
    a.cnt[v] = nc;
    const bool chg = bits_of(old) != bits_of(nv);
    ++nreq;
    nprog += (chg || nc != oc) ? 1u : 0u;
    if (chg) {
        ++nchg;
        if constexpr (sizeof(T) == 8) a.hp[v] = proxy_of(nv);
    }
    return chg;
}

// A list entry's voxel.
struct SweepVoxel {
    bool on;
    uint32_t entry, w;
    int x, y, z;
};
__device__ __forceinline__ SweepVoxel sweep_voxel(const SweepSmem &sm, uint32_t j, uint32_t total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SweepVoxel v;
    v.on = j + lane < total;
    v.entry = v.on ? sm.list[warp][j + lane] : 0u;
    const int4 at = sm.at[warp][v.entry >> 5];
    v.w = static_cast<uint32_t>(at.w);
    v.x = at.x + static_cast<int>(v.entry & 31u);
    v.y = at.y;
    v.z = at.z;
    return v;
}

// Detection of the `total` listed voxels of a warp's 32 words (lane l holds
// word w).  fp64: on the proxies, failed certificates into the warp's buffer
// (ndefer entries), which is decided on full keys 32 at a time; `finish`: to
// the end.  fp32: on the values.  v: fmax, fmin, fdir, active.
template <typename T, class A>
__device__ __forceinline__ void detect_words(SweepSmem &sm, const A &a, const SweepStep *steps, uint32_t *nxt, uint8_t *fnxt,
                                             uint32_t total, uint32_t w, bool finish, uint32_t (&v)[4], uint32_t &ndefer) {
    constexpr bool keys = sizeof(T) == 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SweepBits &bits = sm.bits[warp];
    v[3] += lane == 0 ? total : 0u;
    for (uint32_t j = 0;;) {
        const bool buffered = !keys && (ndefer >= 32 || (finish && ndefer && j >= total));
        if (!buffered && j >= total) break;
        if (!buffered && !keys) {
            const SweepVoxel p = sweep_voxel(sm, j, total);
            const bool inside = p.on && sweep_interior(a.g, p.x, p.y, p.z);
            bool open = p.on;
            const bool all_inside = __all_sync(0xFFFFFFFFu, inside || !p.on);
            if (p.on) {
                const size_t i = flat(a.g, p.x, p.y, p.z);
                const uint8_t c = __ldg(a.codes + i);
                const Ext e = all_inside ? sweep_proxies(a, i) : sweep_proxies_face(a, i, p.x, p.y, p.z);
                open = !e.exact;
                if (!open)
                    sweep_outcome(a, steps, bits, true, nxt, fnxt, p.entry, p.w, e.asc, e.desc, c, v[0], v[1], v[2]);
            }
            const uint32_t md = __ballot_sync(0xFFFFFFFFu, open);
            if (md) {
                if (open)
                    sm.defer[warp][ndefer + static_cast<uint32_t>(__popc(md & ((1u << lane) - 1u)))] =
                        make_uint2(p.w, p.entry & 31u);
                ndefer += static_cast<uint32_t>(__popc(md));
            }
            j += 32;
            continue;
        }
        SweepVoxel p;
        if (buffered) {
            __syncwarp();
            const uint32_t from = ndefer > 32 ? ndefer - 32 : 0;
            p.on = from + lane < ndefer;
            const uint2 e = p.on ? sm.defer[warp][from + lane] : make_uint2(0u, 0u);
            int wx;
            word_coords(a.g, e.x, wx, p.y, p.z);
            p.w = e.x;
            p.entry = e.y;
            p.x = wx * 32 + static_cast<int>(e.y);
            ndefer = from;
            __syncwarp();
        } else {
            p = sweep_voxel(sm, j, total);
            j += 32;
        }
        const bool inside = __all_sync(0xFFFFFFFFu, !p.on || sweep_interior(a.g, p.x, p.y, p.z));
        if (p.on) {
            const size_t i = flat(a.g, p.x, p.y, p.z);
            int asc, desc;
            sweep_keys<T>(a, i, p.x, p.y, p.z, inside, asc, desc);
            sweep_outcome(a, steps, bits, !buffered, nxt, fnxt, p.entry, p.w, asc, desc, __ldg(a.codes + i), v[0],
                          v[1], v[2]);
        }
    }
    __syncwarp();
    const uint32_t own = bits.own[lane];
    if (own) {
        bits.own[lane] = 0;
        atomicOr(nxt + w, own);
        fnxt[w / kGroupWords] = 1;
    }
#pragma unroll
    for (int r = 0; r < kSweepRows; ++r) {
        const uint32_t m = bits.row[r][lane];
        if (m) {
            bits.row[r][lane] = 0;
            const uint32_t wt = w + row_words(a.g, r);
            atomicOr(a.req + wt, m);
            a.freq[wt / kGroupWords] = 1;
        }
    }
}

// The edits of the listed voxels, and the closed stencils of those whose value
// changed.  v: requested, changed, progressed.
template <typename T, class A>
__device__ __forceinline__ void edit_words(SweepSmem &sm, const A &a, uint32_t *nxt, uint8_t *fnxt, uint32_t total,
                                           uint32_t (&v)[4]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t j = 0; j < total; j += 32) {
        const SweepVoxel p = sweep_voxel(sm, j, total);
        uint32_t cb = 0;
        if (p.on && sweep_edit<T>(a, flat(a.g, p.x, p.y, p.z), v[0], v[1], v[2])) cb = 1u << (p.entry & 31u);
        if (cb) atomicOr(&sm.bits[warp].own[p.entry >> 5], cb);
    }
    __syncwarp();
    const uint32_t c = sm.bits[warp].own[lane];
    if (c) {
        sm.bits[warp].own[lane] = 0;
        const int4 at = sm.at[warp][lane];
        mark_words(nxt, fnxt, a.g, static_cast<uint32_t>(at.w), at.x >> 5, at.y, at.z, c);
    }
}

__device__ __forceinline__ void clear_bits(SweepBits &b) {
    const int lane = threadIdx.x & 31;
    b.own[lane] = 0;
    for (int r = 0; r < kSweepRows; ++r) b.row[r][lane] = 0;
    __syncwarp();
}

// The set bits of this lane's word as entries of the warp's list, in order;
// their coordinates into at.  Returns the warp's count.
__device__ __forceinline__ uint32_t list_words(SweepSmem &sm, const Geom &g, uint64_t w, uint32_t word) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (word) {
        int wx, y, z;
        word_coords(g, w, wx, y, z);
        sm.at[warp][lane] = make_int4(wx << 5, y, z, static_cast<int>(static_cast<uint32_t>(w)));
    }
    const uint32_t c = static_cast<uint32_t>(__popc(word));
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += u;
    }
    for (uint32_t p = inc - c; word; word &= word - 1, ++p)
        sm.list[warp][p] = static_cast<uint16_t>((lane << 5) | (__ffs(word) - 1));
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, inc, 31);
    __syncwarp();
    return total;
}

// The flags of a chunk as bits, in one load (one byte after the other, each
// behind the last one's store, cost a chunk of four 1.5 us a phase).  Chunks of
// 1, 2, 4 or 8 start at multiples of their size, and the flags are padded to 256.
__device__ __forceinline__ uint32_t chunk_flags(const uint8_t *p, uint32_t chunk) {
    auto bits = [](uint32_t v) { return ((v * 0x01020408u) >> 24) & 0xFu; };  // bytes of 0 or 1
    if (chunk == 8) {
        const uint2 v = *reinterpret_cast<const uint2 *>(p);
        return bits(v.x) | (bits(v.y) << 4);
    }
    return bits(chunk == 4 ? *reinterpret_cast<const uint32_t *>(p) : chunk == 2 ? *reinterpret_cast<const uint16_t *>(p) : *p);
}
__device__ __forceinline__ void clear_chunk_flags(uint8_t *p, uint32_t chunk) {
    if (chunk == 8) *reinterpret_cast<uint2 *>(p) = make_uint2(0u, 0u);
    else if (chunk == 4) *reinterpret_cast<uint32_t *>(p) = 0;
    else if (chunk == 2) *reinterpret_cast<uint16_t *>(p) = 0;
    else *p = 0;
}

// Calls visit(total, word, last) on the listed set bits of every flagged group
// of this block, up to four groups at a time (lane l holds word l), clearing
// bits and flags; last: this warp's last call.  Chunks of `chunk` neighbouring
// groups are dealt to the warps of the grid in turn: eight (2048 voxels, whose
// stencils share cache lines) where the field has enough of them for every
// thread, fewer in small fields.  The flagged groups of a block's chunks are
// listed in order (blocks then move through the field together, and share its
// cache lines), and its warps take them from the list as they come free.
// RANGE: only the words [lo, hi); a group that reaches beyond them stays flagged.
template <bool RANGE, class Visit>
__device__ __forceinline__ void for_each_group(SweepSmem &sm, uint32_t *bm, uint8_t *flag, const Geom &g, uint32_t chunk,
                                               uint64_t lo, uint64_t hi, Visit &&visit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // groups g0 (a multiple of the chunk) .. ng - 1
    const uint64_t g0 = RANGE ? (lo / kGroupWords) & ~7ull : 0, ng = RANGE ? (hi + kGroupWords - 1) / kGroupWords : group_count(g);
    const uint64_t nc = (ng - g0 + chunk - 1) / chunk;
    for (uint64_t base = 0; base < nc; base += static_cast<uint64_t>(kSweepBlock) * gridDim.x) {
        const uint64_t mine = g0 + (base + static_cast<uint64_t>(threadIdx.x) * gridDim.x + blockIdx.x) * chunk;  // this thread's chunk
        uint32_t fm = 0;
        if (mine < ng) {
            fm = chunk_flags(flag + mine, chunk);
            if (RANGE) {  // the groups of the range, and of these the ones inside it
                uint32_t in = 0, inside = 0;
                for (uint32_t j = 0; j < chunk; ++j) {
                    const uint64_t w0 = (mine + j) * kGroupWords;
                    in |= (w0 + kGroupWords > lo && w0 < hi ? 1u : 0u) << j;
                    inside |= (w0 >= lo && w0 + kGroupWords <= hi ? 1u : 0u) << j;
                }
                fm &= in;
                for (uint32_t m = fm & inside; m; m &= m - 1) flag[mine + static_cast<uint32_t>(__ffs(m) - 1)] = 0;
            } else if (fm) {
                clear_chunk_flags(flag + mine, chunk);
            }
        }
        const uint32_t c = static_cast<uint32_t>(__popc(fm));
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) sm.groups[warp] = inc;
        if (threadIdx.x == 0) sm.next = 0;
        __syncthreads();
        uint32_t first = inc - c, groups = 0;
#pragma unroll
        for (int k = 0; k < kSweepWarps; ++k) {
            const uint32_t n = sm.groups[k];
            first += k < warp ? n : 0u;
            groups += n;
        }
        for (; fm; fm &= fm - 1, ++first) sm.group[first] = static_cast<uint16_t>(threadIdx.x * 8 + __ffs(fm) - 1);
        __syncthreads();
        // as few rounds of up to four as it takes, then as evenly as they come
        const uint32_t rounds = (groups + 4 * kSweepWarps - 1) / (4 * kSweepWarps);
        const uint32_t take = groups ? (groups + kSweepWarps * rounds - 1) / (kSweepWarps * rounds) : 1u;
        auto next_words = [&](uint64_t &w) -> uint32_t {  // this lane's word of the next groups (none: w = ~0 in every lane)
            uint32_t t = lane == 0 ? atomicAdd(&sm.next, take) : 0u;
            t = __shfl_sync(0xFFFFFFFFu, t, 0);
            w = ~0ull;
            const uint32_t i = lane >> 3;
            if (i < take && t + i < groups) {
                const uint32_t e = sm.group[t + i];
                w = (g0 + (base + static_cast<uint64_t>(e >> 3) * gridDim.x + blockIdx.x) * chunk + (e & 7u)) *
                        kGroupWords + (lane & 7);
            }
            return (RANGE ? w >= lo && w < hi : w < g.nwords) ? bm[w] : 0u;
        };
        uint64_t w;
        uint32_t word = next_words(w);
        while (__shfl_sync(0xFFFFFFFFu, w, 0) != ~0ull) {
            uint64_t w_next;
            const uint32_t next = next_words(w_next);  // in flight while these groups are visited
            if (word) bm[w] = 0;
            const uint32_t total = list_words(sm, g, w, word);
            visit(total, static_cast<uint32_t>(w), __shfl_sync(0xFFFFFFFFu, w_next, 0) == ~0ull);
            __syncwarp();  // list and at are rewritten by the next groups
            w = w_next;
            word = next;
        }
        __syncthreads();  // group, groups and next are rewritten by the next chunks
    }
}

template <typename T>
__global__ void __launch_bounds__(kSweepBlock, 3) k_sweeps(const __grid_constant__ SweepArgs<T> a) {
    __shared__ SweepSmem sm;
    uint32_t target = 0;  // of the grid barrier
    const Geom &g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t chunk = 8;
    while (chunk > 1 && group_count(g) < static_cast<uint64_t>(chunk) * gridDim.x * kSweepWarps) chunk >>= 1;
    if (warp == 0) fill_steps(sm.step, g, lane);
    clear_bits(sm.bits[warp]);
    __syncthreads();
    int64_t k = 0;
    bool edits_only = a.from_edits != 0;
    if (!edits_only) {  // every block reads the same state: all return, or none
        k = a.ls->k;
        if (!a.ls->go) {
            if (blockIdx.x == 0 && threadIdx.x == 0) a.ls->done = k;
            return;
        }
    }
    while (true) {
        uint32_t *cur = (k & 1) ? a.act1 : a.act0, *nxt = (k & 1) ? a.act0 : a.act1;
        uint8_t *fcur = (k & 1) ? a.f1 : a.f0, *fnxt = (k & 1) ? a.f0 : a.f1;
        if (!edits_only) {
            const SweepSlot *p = a.slots + (k - 1);
            if (sweep_stops(p->fmax, p->fmin, p->fdir, p->progressed, k, a.max_sweeps) || (k == 1 && p->bad)) break;
            uint32_t c[4] = {0u, 0u, 0u, 0u}, ndefer = 0;
            for_each_group<false>(sm, cur, fcur, g, chunk, 0, 0, [&](uint32_t total, uint32_t w, bool last) {
                detect_words<T>(sm, a, sm.step, nxt, fnxt, total, w, last, c, ndefer);
            });
            const uint32_t v[8] = {c[0], c[1], c[2], 0u, 0u, 0u, c[3], 0u};
            block_flush_slot(a.slots + k, v);
            if (!sweep_barrier(&a.ls->bar[0], target, &a.ls->err)) return;
        }
        edits_only = false;
        {
            uint32_t c[4] = {0u, 0u, 0u, 0u};
            for_each_group<false>(sm, a.req, a.freq, g, chunk, 0, 0,
                           [&](uint32_t total, uint32_t, bool) { edit_words<T>(sm, a, nxt, fnxt, total, c); });
            const uint32_t v[8] = {0u, 0u, 0u, c[0], c[1], c[2], 0u, 0u};
            block_flush_slot(a.slots + k, v);
        }
        if (!sweep_barrier(&a.ls->bar[0], target, &a.ls->err)) return;
        ++k;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ls->done = k;
}

// The sweeps behind the host copy (first_pass_waves): in one launch, on the
// planes that are final so far, the pieces of sweeps 0 .. K that these planes
// allow: of sweep k the detection of words [det0, det1) and then the edits of
// words [edit0, edit1), every piece behind a grid barrier.  The counters add up
// in the sweeps' slots over the launches.
constexpr int kWaveSweeps = 6;
struct WaveFronts {  // words: the fronts of the launch before and of this one
    uint32_t det0[kWaveSweeps + 1], det1[kWaveSweeps + 1], edit0[kWaveSweeps + 1], edit1[kWaveSweeps + 1];
    int sweeps;             // K
    int launch;             // its barrier counter, 1 ..
};
template <typename T>
__global__ void __launch_bounds__(kSweepBlock, 3) k_sweep_wave(const __grid_constant__ SweepArgs<T> a,
                                                               const __grid_constant__ WaveFronts f) {
    __shared__ SweepSmem sm;
    uint32_t target = 0;  // of the grid barrier
    const Geom &g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) fill_steps(sm.step, g, lane);
    clear_bits(sm.bits[warp]);
    __syncthreads();
    auto chunk_of = [&](uint32_t words) {
        uint32_t chunk = 8;
        while (chunk > 1 && words / kGroupWords < static_cast<uint64_t>(chunk) * gridDim.x * kSweepWarps) chunk >>= 1;
        return chunk;
    };
    for (int k = 0; k <= f.sweeps; ++k) {
        uint32_t *cur = (k & 1) ? a.act1 : a.act0, *nxt = (k & 1) ? a.act0 : a.act1;
        uint8_t *fcur = (k & 1) ? a.f1 : a.f0, *fnxt = (k & 1) ? a.f0 : a.f1;
        if (k > 0 && f.det1[k] > f.det0[k]) {  // (of sweep 0 the first pass is the detection)
            uint32_t c[4] = {0u, 0u, 0u, 0u}, ndefer = 0;
            for_each_group<true>(sm, cur, fcur, g, chunk_of(f.det1[k] - f.det0[k]), f.det0[k], f.det1[k],
                                 [&](uint32_t total, uint32_t w, bool last) {
                                     detect_words<T>(sm, a, sm.step, nxt, fnxt, total, w, last, c, ndefer);
                                 });
            const uint32_t v[8] = {c[0], c[1], c[2], 0u, 0u, 0u, c[3], 0u};
            block_flush_slot(a.slots + k, v);
            if (!sweep_barrier(&a.ls->bar[f.launch], target, &a.ls->err)) return;
        }
        if (f.edit1[k] > f.edit0[k]) {
            uint32_t c[4] = {0u, 0u, 0u, 0u};
            for_each_group<true>(sm, a.req, a.freq, g, chunk_of(f.edit1[k] - f.edit0[k]), f.edit0[k], f.edit1[k],
                                 [&](uint32_t total, uint32_t, bool) { edit_words<T>(sm, a, nxt, fnxt, total, c); });
            const uint32_t v[8] = {0u, 0u, 0u, c[0], c[1], c[2], 0u, 0u};
            block_flush_slot(a.slots + k, v);
            if (!sweep_barrier(&a.ls->bar[f.launch], target, &a.ls->err)) return;
        }
    }
}

// After the wavefront has run sweeps 0 .. K to the end: the state after sweep
// K, or after the first of those sweeps that stops the loop (the sweeps after a
// stopping one changed nothing: they found an empty active set, or repeated a
// sweep whose edits changed no value and no counter, or follow a NaN input
// whose call fails).
static __global__ void k_wave_gate(LoopState *ls, const SweepSlot *slots, long long K, long long max_sweeps) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    long long k = 0;
    bool stop = false;
    for (; k <= K; ++k) {
        const SweepSlot c = slots[k];
        stop = (k == 0 && c.bad) || sweep_stops(c.fmax, c.fmin, c.fdir, c.progressed, k + 1, max_sweeps);
        if (stop) break;
    }
    ls->k = stop ? k + 1 : K + 1;
    ls->go = stop ? 0 : 1;
}

}  // namespace pmsz
