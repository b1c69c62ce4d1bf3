// tiled.cuh -- the proxies that the stencil kernels compare (march.cuh and
// sweep.cuh include this file), and the edits of full sweeps.
//
// GB300 executes integer compare / min / max (and FP32 min / max) on one
// 64-lane-per-clock pipe per SM, so a 15-point argmax / argmin on 64-bit keys
// (about five instructions per candidate) would bound the sweeps, not HBM.
// They compare 32-bit PROXIES instead:
//
//   proxy(v) = the high 28 bits of an order-preserving key, low 4 bits clear
//
// so that `proxy + rank` packs a candidate's stencil rank into the free bits
// and a whole argmax is one min/max instruction per candidate.  Truncation
// can only merge keys, never reorder them (key_a < key_b => proxy_a <=
// proxy_b), so the packed chain is exact whenever the winning proxy is
// unique.  A second chain with the ranks reversed (15 - r) picks the LOWEST
// rank among tied proxies; both chains agree exactly when the winner is
// unique -- the exactness certificate.  Where they disagree (ties in the
// truncated proxy) the voxel takes the exact path on full keys.  (march.cuh packs
// tags of the coordinates instead of ranks.)
//
// Out-of-domain stencil cells hold proxy 0: as `0 + r` they lose every max
// chain (real proxies are >= 16), and the min chains add -16 (or -1) so that
// they wrap to the top of the range and lose every min chain; no per-lane
// boundary branch is needed on the fast path.
#pragma once
#include <cuda.h>  // CUtensorMap (the map itself is encoded on the host)

#include "helpers.cuh"

namespace pmsz {

// The proxy of a value: 0x80000000 plus or minus the top 31 magnitude bits,
// low 4 bits cleared.  Monotone in the value, and -0 and +0 coincide, with no
// test for zero (fp64: negative magnitudes are truncated towards zero, so the
// proxy is not the high word of okey, only ordered the same way).
__device__ __forceinline__ uint32_t proxy_of_bits(uint32_t hi) {
    const uint32_t s = static_cast<uint32_t>(static_cast<int32_t>(hi) >> 31);
    return (((hi & 0x7FFFFFFFu) ^ s) - s + 0x80000000u) & ~15u;
}
__device__ __forceinline__ uint32_t proxy_of(double v) { return proxy_of_bits(static_cast<uint32_t>(__double2hiint(v))); }
__device__ __forceinline__ uint32_t proxy_of(float v) { return proxy_of_bits(__float_as_uint(v)); }

struct Ext {
    int asc, desc;
    bool exact;
};

// Packed argmax / argmin of 15 proxies in rank order, with certificates.
// General form: out-of-domain candidates carry proxy 0; the min chains add
// -16 (and -1) so those wrap to the top of the range and lose.  Each chain step
// is one fused add-and-max / add-and-min (__viaddmax_u32 / __viaddmin_u32:
// max(a + b, c), min(a + b, c), 32-bit wrapping add).
__device__ __forceinline__ Ext proxy_ext(const uint32_t (&t)[15]) {
    uint32_t M = t[0], M2 = t[0] + 15u, m = t[0] - 16u, m2 = t[0] - 1u;
#pragma unroll
    for (int r = 1; r < 15; ++r) {
        M = __viaddmax_u32(t[r], static_cast<uint32_t>(r), M);
        M2 = __viaddmax_u32(t[r], static_cast<uint32_t>(15 - r), M2);
        m = __viaddmin_u32(t[r], static_cast<uint32_t>(r) - 16u, m);
        m2 = __viaddmin_u32(t[r], 0u - 1u - static_cast<uint32_t>(r), m2);
    }
    Ext e;
    e.asc = static_cast<int>(M & 15u);
    e.desc = static_cast<int>(m & 15u);
    e.exact = e.asc == 15 - static_cast<int>(M2 & 15u) && e.desc == 15 - static_cast<int>(m2 & 15u);
    return e;
}

// Interior form (all 15 candidates inside the domain): the max and min chains
// take the same packed values t + r and t + (15 - r).
__device__ __forceinline__ Ext proxy_ext_interior(const uint32_t (&t)[15]) {
    uint32_t M = t[0], m = t[0], M2 = t[0] + 15u, m2 = M2;
#pragma unroll
    for (int r = 1; r < 15; ++r) {
        M = __viaddmax_u32(t[r], static_cast<uint32_t>(r), M);
        m = __viaddmin_u32(t[r], static_cast<uint32_t>(r), m);
        M2 = __viaddmax_u32(t[r], static_cast<uint32_t>(15 - r), M2);
        m2 = __viaddmin_u32(t[r], static_cast<uint32_t>(15 - r), m2);
    }
    Ext e;
    e.asc = static_cast<int>(M & 15u);
    e.desc = static_cast<int>(m & 15u);
    e.exact = e.asc == 15 - static_cast<int>(M2 & 15u) && e.desc == 15 - static_cast<int>(m2 & 15u);
    return e;
}

constexpr int kHX = kTX + 2;
constexpr int kThreads = kTX * kMY / 2;
// ---------------------------------------------------------------------------
// Block-local compaction of a bitmap.  A round covers 2048 consecutive words:
// each of the 256 threads loads 8 of them with two 16-byte loads, and one
// barrier skips the round when all are empty (late sweeps touch a few words of
// a large bitmap, so the scan must move as much per barrier as it can).  In a
// non-empty round the set bits of all 2048 words are ranked by a block scan
// and written to a dense work list in shared memory (entries (word << 5) |
// bit, word local to the round), in passes of at most kListCap entries, and
// all 256 threads share the list: a sparse or clustered bitmap still keeps
// every lane busy, and a sparse round costs a handful of barriers.
// ---------------------------------------------------------------------------
constexpr int kListBlock = 256;
constexpr int kWordsPerThread = 8;
constexpr int kRoundWords = kListBlock * kWordsPerThread;
constexpr uint32_t kListCap = 8192;

struct ListSmem {
    uint32_t list[kListCap];
    uint32_t warp_tot[kListBlock / 32];
    uint32_t total;
};

// Loads the 8 words of this thread for the round starting at `base` (bitmaps
// are 256-byte aligned and rounds start at multiples of 2048 words, so the
// vector loads are aligned); returns whether any word of the block is set.
__device__ __forceinline__ bool load_round(const uint32_t *__restrict__ bm, size_t base, const Geom &g,
                                           uint32_t (&w8)[kWordsPerThread]) {
    const size_t w0 = base + static_cast<size_t>(threadIdx.x) * kWordsPerThread;
    if (w0 + kWordsPerThread <= g.nwords) {
        const uint4 a = __ldg(reinterpret_cast<const uint4 *>(bm + w0));
        const uint4 b = __ldg(reinterpret_cast<const uint4 *>(bm + w0 + 4));
        w8[0] = a.x; w8[1] = a.y; w8[2] = a.z; w8[3] = a.w;
        w8[4] = b.x; w8[5] = b.y; w8[6] = b.z; w8[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < kWordsPerThread; ++j) w8[j] = w0 + j < g.nwords ? __ldg(bm + w0 + j) : 0u;
    }
    uint32_t any = 0;
#pragma unroll
    for (int j = 0; j < kWordsPerThread; ++j) any |= w8[j];
    return __syncthreads_or(any != 0) != 0;
}

// Calls work(x, y, z) for every set bit of bitmap `bm` (clearing the bitmap).
// Every thread of the block must call this.
// One round (2048 words from `base`) of for_each_set_bit.
template <class Work>
__device__ __forceinline__ void process_round(ListSmem &sm, uint32_t *__restrict__ bm, const Geom &g, size_t base,
                                              Work &work) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    {
        uint32_t w8[kWordsPerThread];
        if (!load_round(bm, base, g, w8)) return;  // uniform
        const size_t w0 = base + static_cast<size_t>(t) * kWordsPerThread;
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < kWordsPerThread; ++j) {
            if (w8[j]) bm[w0 + j] = 0;
            c += __popc(w8[j]);
        }
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) sm.warp_tot[warp] = inc;
        __syncthreads();
        if (t == 0) {
            uint32_t run = 0;
            for (int k = 0; k < kListBlock / 32; ++k) {
                const uint32_t v = sm.warp_tot[k];
                sm.warp_tot[k] = run;
                run += v;
            }
            sm.total = run;
        }
        __syncthreads();
        const uint32_t first = sm.warp_tot[warp] + inc - c, total = sm.total;
        for (uint32_t lo = 0; lo < total; lo += kListCap) {
            const uint32_t hi = lo + kListCap;
            if (first < hi && first + c > lo) {  // some of my entries fall in this pass
                uint32_t rank = first;
#pragma unroll
                for (int j = 0; j < kWordsPerThread; ++j) {
                    uint32_t bits = w8[j];
                    while (bits) {
                        const int b = __ffs(bits) - 1;
                        bits &= bits - 1;
                        if (rank >= lo && rank < hi)
                            sm.list[rank - lo] = (static_cast<uint32_t>(t * kWordsPerThread + j) << 5) | static_cast<uint32_t>(b);
                        ++rank;
                    }
                }
            }
            __syncthreads();
            const uint32_t n = min(kListCap, total - lo);
            for (uint32_t k = t; k < n; k += kListBlock) {
                const uint32_t e = sm.list[k];
                const uint32_t wl = e >> 5;
                const int b = static_cast<int>(e & 31u);
                int wx, y, z;
                word_coords(g, base + wl, wx, y, z);
                work(wx * 32 + b, y, z);
            }
            __syncthreads();
        }
    }
}

template <class Work>
__device__ __forceinline__ void for_each_set_bit(ListSmem &sm, uint32_t *__restrict__ bm, const Geom &g, Work &work) {
    for (size_t base = static_cast<size_t>(blockIdx.x) * kRoundWords; base < g.nwords;
         base += static_cast<size_t>(gridDim.x) * kRoundWords)
        process_round(sm, bm, g, base, work);
}

// ---------------------------------------------------------------------------
// The edits of a full sweep: applyDeltaBuffer_local (pMSz.cu:623-645) on
// every requested vertex, in T:
//   if |f - (fhat - delta)| <= eps && cnt < q-1 { fhat -= delta; cnt++ }
//   else { cnt = q; fhat = f - eps }
// (The next full sweep looks at every voxel: no active set, no proxies.)
// ---------------------------------------------------------------------------
template <typename T>
struct ApplyWork {
    const T *f;
    T *fh;
    uint8_t *cnt;
    Geom g;
    T eps, delta;
    int q;
    uint32_t nreq = 0, nchg = 0, nprog = 0;
    __device__ __forceinline__ void operator()(int x, int y, int z) {
        bool progressed;
        nchg += apply_one(f, fh, cnt, flat(g, x, y, z), eps, delta, q, progressed);
        ++nreq;
        nprog += progressed ? 1u : 0u;
    }
};

template <typename T>
__global__ void __launch_bounds__(kListBlock) k_apply_full(const T *__restrict__ f, T *__restrict__ fh,
                                                           uint8_t *__restrict__ cnt, uint32_t *__restrict__ req,
                                                           SweepSlot *slot, Geom g, T eps, T delta, int q) {
    __shared__ ListSmem sm;
    ApplyWork<T> work{f, fh, cnt, g, eps, delta, q};
    for_each_set_bit(sm, req, g, work);
    const uint32_t v[8] = {0u, 0u, 0u, work.nreq, work.nchg, work.nprog, 0u, 0u};
    block_flush_slot(slot, v);
}

// Stop rule of the correction loop after a sweep (the slot of that sweep):
// converged (no mismatch), stuck (nothing could change), or out of sweeps.
__host__ __device__ __forceinline__ bool sweep_stops(unsigned long long fmax, unsigned long long fmin,
                                                     unsigned long long fdir, unsigned long long progressed,
                                                     int64_t sweeps_done, int64_t max_sweeps) {
    return (fmax == 0 && fmin == 0 && fdir == 0) || progressed == 0 || sweeps_done >= max_sweeps;
}

}  // namespace pmsz
