// sweep.cuh -- the correction loop's sweeps in one cooperative launch, included
// by correct.cu after list.cuh.
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
//  * Chunks of groups are dealt round-robin to all warps of the grid,
//    neighbouring chunks to different SMs, so a cluster of activity spreads over
//    the chip.
//  * A warp takes four flagged groups at a time, lists their set bits in shared
//    memory (each lane the bits of its own word at its prefix), then visits them
//    32 at a time: nearly full warps whatever the density, and no barrier wider
//    than the warp.
//  * Loads are ordinary cached loads: a grid barrier orders them behind the
//    other blocks' writes, and within a phase no array is both read at
//    neighbours and written (detection reads proxies and codes and writes
//    bitmaps, the edits touch their own voxel's values only), so the 15 gathers
//    of neighbouring voxels share L1 lines.
//  * Failed certificates collect in a per-warp buffer and are decided on full
//    keys 32 at a time; fp32 fields with many (plateaus) detect on exact keys
//    throughout.
//
// Bound by the latency of the gathers and, in small fields and late sweeps, of
// the two grid barriers a sweep takes (about 2 us each).  Three blocks per SM:
// with four (64 registers) fp64 detection is 2 % and dense fp32 sweeps on full
// keys 5 % slower; blocks of 128 threads, five or six blocks per SM, groups of
// 32 words and results merged in shared memory before the marks were all slower.
// Whole corrections, list kernels in a conditional CUDA graph (before) -> this:
//   64^3 fp32, 8 sweeps              358 -> 181 us
//   173x141x203 fp32, 12 sweeps      560 -> 353 us
//   512^3 fp64, 16 sparse sweeps    4134 -> 3654 us (first pass 1.50 -> 1.19 ms of it)
//   256^3 fp32, 27 dense sweeps     4727 -> 4467 us (on full keys)
#pragma once
#include "list.cuh"

namespace pmsz {

constexpr int kSweepBlock = 256, kSweepWarps = kSweepBlock / 32;
constexpr uint32_t kSweepDefer = 64;  // failed certificates buffered per warp (decided from 32 on)

__host__ __device__ __forceinline__ size_t group_count(const Geom &g) {
    return (g.nwords + kGroupWords - 1) / kGroupWords;
}

// or_word / mark_stencil / request_targets that also set the group's flag.
__device__ __forceinline__ void or_word_f(uint32_t *act, uint8_t *flag, const Geom &g, int wx, int y, int z, uint32_t m) {
    if (!m || wx < 0 || wx >= g.wpr || y < 0 || y >= g.ny || z < 0 || z >= g.nz) return;
    m &= row_tail_mask(g, wx);
    if (!m) return;
    const size_t w = static_cast<size_t>(wx) + static_cast<size_t>(g.wpr) * (static_cast<size_t>(y) + static_cast<size_t>(g.ny) * z);
    atomicOr(act + w, m);
    flag[w / kGroupWords] = 1;
}
__device__ __forceinline__ void mark_stencil_f(uint32_t *act, uint8_t *flag, const Geom &g, int wx, int y, int z,
                                               uint32_t c) {
    const uint32_t lo = (c & 1u) << 31, hi = c >> 31;
    or_word_f(act, flag, g, wx, y, z, c | (c << 1) | (c >> 1));
    or_word_f(act, flag, g, wx - 1, y, z, lo);
    or_word_f(act, flag, g, wx + 1, y, z, hi);
    const uint32_t m = c | (c >> 1), p = c | (c << 1);
    or_word_f(act, flag, g, wx, y + 1, z, m);     or_word_f(act, flag, g, wx - 1, y + 1, z, lo);
    or_word_f(act, flag, g, wx, y, z + 1, m);     or_word_f(act, flag, g, wx - 1, y, z + 1, lo);
    or_word_f(act, flag, g, wx, y + 1, z + 1, m); or_word_f(act, flag, g, wx - 1, y + 1, z + 1, lo);
    or_word_f(act, flag, g, wx, y - 1, z, p);     or_word_f(act, flag, g, wx + 1, y - 1, z, hi);
    or_word_f(act, flag, g, wx, y, z - 1, p);     or_word_f(act, flag, g, wx + 1, y, z - 1, hi);
    or_word_f(act, flag, g, wx, y - 1, z - 1, p); or_word_f(act, flag, g, wx + 1, y - 1, z - 1, hi);
}

// The same for the lanes of a warp that each hold a word's merged changed bits
// (lead: this lane does; every lane calls it).  Few words -- runs of changed
// voxels, as in dense sweeps -- take one word after the other, its 14 marks on
// 14 lanes: 40 instructions a word, where one lane's 14 marks in a row are 350.
__device__ __forceinline__ void mark_stencils(uint32_t *act, uint8_t *flag, const Geom &g, bool lead, int wx, int y, int z,
                                              uint32_t c) {
    uint32_t m = __ballot_sync(0xFFFFFFFFu, lead);
    if (__popc(m) > 4) {
        if (lead) mark_stencil_f(act, flag, g, wx, y, z, c);
        return;
    }
    // lane l < 14: the row (dy, dz) of l / 2, and its own word (even) or the
    // neighbouring one that the row's shifted bits reach (odd)
    const int lane = threadIdx.x & 31, row = lane >> 1;
    const int dy = row == 1 || row == 3 ? 1 : row == 4 || row == 6 ? -1 : 0;
    const int dz = row == 2 || row == 3 ? 1 : row == 5 || row == 6 ? -1 : 0;
    // rows 1-3 take x-1, x; rows 4-6 take x, x+1; row 0 takes all three (its
    // second neighbour word is lane 14's)
    const bool left = row == 0 || (row >= 1 && row <= 3), right = row == 0 || (row >= 4 && row <= 6) || lane == 14;
    for (; m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const uint32_t cb = __shfl_sync(0xFFFFFFFFu, c, src);
        const int bx = __shfl_sync(0xFFFFFFFFu, wx, src), by = __shfl_sync(0xFFFFFFFFu, y, src),
                  bz = __shfl_sync(0xFFFFFFFFu, z, src);
        if (lane < 15) {
            const uint32_t lo = (cb & 1u) << 31, hi = cb >> 31;
            uint32_t bits;
            int ox = 0;
            if (lane == 14) {
                bits = hi;
                ox = 1;
            } else if (lane & 1) {
                bits = left ? lo : hi;
                ox = left ? -1 : 1;
            } else {
                bits = cb | (left ? cb >> 1 : 0u) | (right ? cb << 1 : 0u);
            }
            or_word_f(act, flag, g, bx + ox, lane == 14 ? by : by + dy, lane == 14 ? bz : bz + dz, bits);
        }
    }
}

// Flags of a plain bitmap: act0 (f0) or act1 (f1), the one of sweep *k_at.
static __global__ void __launch_bounds__(256) k_build_flags(const uint32_t *act0, const uint32_t *act1, Geom g, uint8_t *f0,
                                                     uint8_t *f1, const long long *k_at) {
    const bool odd = (*k_at & 1) != 0;
    const uint32_t *bm = odd ? act1 : act0;
    uint8_t *flag = odd ? f1 : f0;
    // one thread per word; the lanes of a group vote
    const size_t n = group_count(g) * kGroupWords, step = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t w = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; w - (threadIdx.x & 31) < n; w += step) {
        const uint32_t any = __ballot_sync(0xFFFFFFFFu, w < g.nwords && bm[w] != 0);
        const uint32_t first = (threadIdx.x & 31) & ~(kGroupWords - 1);
        if (w < n && w % kGroupWords == 0) flag[w / kGroupWords] = (any >> first) & ((1u << kGroupWords) - 1u) ? 1 : 0;
    }
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
    uint32_t group[kSweepWarps][256];     // flagged groups to visit
    uint16_t list[kSweepWarps][1024];     // lane of the word << 5 | bit of four groups' set bits
    int4 at[kSweepWarps][32];             // x of bit 0, y, z of their words, and the word
    uint2 defer[kSweepWarps][kSweepDefer];  // word, bit
    uint32_t deferred;
};

// Calls visit(active, word, bit, x, y, z) for the set bits of every flagged
// group of this warp, whole warps at a time (active: the lane has a voxel),
// clearing bits and flags.  Chunks of `chunk` neighbouring groups are dealt to
// the warps in turn: eight (2048 voxels, whose stencils share cache lines) where
// the field has enough of them for every warp, fewer in small fields.
template <class Visit>
__device__ __forceinline__ void for_each_group(SweepSmem &sm, uint32_t *bm, uint8_t *flag, const Geom &g, uint32_t chunk,
                                               Visit &&visit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t W = gridDim.x * kSweepWarps, wid = static_cast<uint32_t>(warp) * gridDim.x + blockIdx.x;
    const uint64_t ng = group_count(g), nc = (ng + chunk - 1) / chunk;
    for (uint64_t base = 0; base < nc; base += 32ull * W) {
        const uint64_t mine = (base + static_cast<uint64_t>(lane) * W + wid) * chunk;  // this lane's chunk
        uint32_t fm = 0;
        if (mine < ng) {  // (the flags are padded to 256 bytes and start at a multiple of the chunk)
            if (chunk == 8) {
                const uint2 v = *reinterpret_cast<const uint2 *>(flag + mine);
                if (v.x | v.y) *reinterpret_cast<uint2 *>(flag + mine) = make_uint2(0u, 0u);
                fm = (((v.x * 0x01020408u) >> 24) & 0xFu) | (((v.y * 0x01020408u) >> 20) & 0xF0u);  // bytes of 0 or 1 -> bits
            } else {
                for (uint32_t j = 0; j < chunk && mine + j < ng; ++j)
                    if (flag[mine + j]) {
                        flag[mine + j] = 0;
                        fm |= 1u << j;
                    }
            }
        }
        const uint32_t c = static_cast<uint32_t>(__popc(fm));
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += v;
        }
        const uint32_t groups = __shfl_sync(0xFFFFFFFFu, inc, 31);
        if (!groups) continue;
        for (uint32_t p = inc - c; fm; fm &= fm - 1, ++p)
            sm.group[warp][p] = static_cast<uint32_t>(mine) + static_cast<uint32_t>(__ffs(fm) - 1);
        __syncwarp();
        auto word_at = [&](uint32_t t) -> uint64_t {  // this lane's word of the four groups from t on
            return t + (lane >> 3) < groups ? static_cast<uint64_t>(sm.group[warp][t + (lane >> 3)]) * kGroupWords + (lane & 7)
                                            : ~0ull;
        };
        uint64_t w = word_at(0);
        uint32_t word = w < g.nwords ? bm[w] : 0u;
        for (uint32_t t = 0; t < groups; t += 4) {
            const uint64_t w_next = word_at(t + 4);
            const uint32_t next = w_next < g.nwords ? bm[w_next] : 0u;  // in flight while these groups are visited
            if (word) {
                bm[w] = 0;
                int wx, y, z;
                word_coords(g, w, wx, y, z);
                sm.at[warp][lane] = make_int4(wx << 5, y, z, static_cast<int>(static_cast<uint32_t>(w)));
            }
            const uint32_t cw = static_cast<uint32_t>(__popc(word));
            uint32_t iw = cw;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, iw, o);
                if (lane >= o) iw += v;
            }
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, iw, 31);
            for (uint32_t p = iw - cw; word; word &= word - 1, ++p)
                sm.list[warp][p] = static_cast<uint16_t>((lane << 5) | (__ffs(word) - 1));
            __syncwarp();
            for (uint32_t j = 0; j < total; j += 32) {
                const bool on = j + lane < total;
                const uint32_t e = on ? sm.list[warp][j + lane] : 0u;
                const int4 at = on ? sm.at[warp][e >> 5] : make_int4(0, 0, 0, 0);
                visit(on, static_cast<uint32_t>(at.w), static_cast<int>(e & 31u), at.x + static_cast<int>(e & 31u), at.y,
                      at.z);
            }
            __syncwarp();  // list and at are rewritten by the next groups
            w = w_next;
            word = next;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kSweepBlock, 3) k_sweeps(const __grid_constant__ SweepArgs<T> a) {
    __shared__ SweepSmem sm;
    cg::grid_group grid = cg::this_grid();
    const Geom &g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const ptrdiff_t sy = g.nx, sz = static_cast<ptrdiff_t>(g.nx) * g.ny;
    uint32_t chunk = 8;
    while (chunk > 1 && group_count(g) < static_cast<uint64_t>(chunk) * 8u * gridDim.x * kSweepWarps) chunk >>= 1;
    int64_t k = 0;
    bool edits_only = a.from_edits != 0;
    if (!edits_only) {  // every block reads the same state: all return, or none
        k = a.ls->k;
        if (!a.ls->go) {
            if (blockIdx.x == 0 && threadIdx.x == 0) a.ls->done = k;
            return;
        }
    }
    // fp32: exact keys when the first pass decided more than a tenth of the
    // voxels on keys, or a sweep did (for good)
    bool keys = sizeof(T) == 4 && 10ull * a.ls->lc[3] > static_cast<unsigned long long>(g.n);
    while (true) {
        uint32_t *cur = (k & 1) ? a.act1 : a.act0, *nxt = (k & 1) ? a.act0 : a.act1;
        uint8_t *fcur = (k & 1) ? a.f1 : a.f0, *fnxt = (k & 1) ? a.f0 : a.f1;
        if (!edits_only) {
            const SweepSlot *p = a.slots + (k - 1);
            if (sweep_stops(p->fmax, p->fmin, p->fdir, p->progressed, k, a.max_sweeps) || (k == 1 && p->bad)) break;
            uint32_t cmax = 0, cmin = 0, cdir = 0, active = 0, ndefer = 0, ndeferred = 0;
            if (threadIdx.x == 0) sm.deferred = 0;
            auto outcome = [&](uint32_t w, int bit, int x, int y, int z, int asc, int desc, uint8_t c) {
                uint32_t tm = detect_rules(asc, desc, c & 15, c >> 4, cmax, cmin, cdir);
                if (!tm) return;
                atomicOr(nxt + w, 1u << bit);
                fnxt[w / kGroupWords] = 1;
                for (; tm; tm &= tm - 1) {
                    const uint32_t r2 = 2u * static_cast<uint32_t>(__ffs(tm) - 1);
                    const int tx = x + static_cast<int>((kStepX >> r2) & 3u) - 1,
                              ty = y + static_cast<int>((kStepY >> r2) & 3u) - 1,
                              tz = z + static_cast<int>((kStepZ >> r2) & 3u) - 1;
                    const size_t wt = word_of(g, tx, ty, tz);
                    atomicOr(a.req + wt, 1u << (tx & 31));
                    a.freq[wt / kGroupWords] = 1;
                }
            };
            // Full keys of one voxel (interior: of a warp whose voxels all are).
            auto on_keys = [&](uint32_t w, int bit, int x, int y, int z, bool interior) {
                const size_t i = flat(g, x, y, z);
                const T *c0 = a.fh + i;
                using K = typename KeyOf<T>::type;
                constexpr int kKeyLoads = 5;  // in flight (fp64 keys are two registers each; fp32 is no faster with 15)
                K hi = 0, lo = ~K(0);
                int asc = kSelf, desc = kSelf;
                auto scan = [&](auto test) {
#pragma unroll
                    for (int r0 = 0; r0 < 15; r0 += kKeyLoads) {
                        K kk[kKeyLoads];
#pragma unroll
                        for (int j = 0; j < kKeyLoads; ++j) {
                            const int r = r0 + j;
                            kk[j] = test(r) ? okey(c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz]) : K(0);
                        }
#pragma unroll
                        for (int j = 0; j < kKeyLoads; ++j)
                            if (test(r0 + j)) {
                                if (kk[j] >= hi) { hi = kk[j]; asc = r0 + j; }
                                if (kk[j] < lo) { lo = kk[j]; desc = r0 + j; }
                            }
                    }
                };
                if (interior) {
                    scan([](int) { return true; });
                } else {
                    const uint32_t valid = valid_mask(x, y, z, g.nx, g.ny, g.nz);
                    scan([&](int r) { return ((valid >> r) & 1u) != 0; });
                }
                outcome(w, bit, x, y, z, asc, desc, __ldg(a.codes + i));
            };
            auto drain = [&](uint32_t from, uint32_t to) {  // buffered voxels, one per lane
                __syncwarp();
                if (from + lane < to) {
                    const uint2 e = sm.defer[warp][from + lane];
                    int wx, y, z;
                    word_coords(g, e.x, wx, y, z);
                    on_keys(e.x, static_cast<int>(e.y), wx * 32 + static_cast<int>(e.y), y, z, false);
                }
                __syncwarp();
            };
            for_each_group(sm, cur, fcur, g, chunk, [&](bool on, uint32_t w, int bit, int x, int y, int z) {
                bool exact = true;
                // nearly every warp has only interior voxels: no test per gather
                const bool inside = x >= 1 && x <= g.nx - 2 && y >= 1 && y <= g.ny - 2 && z >= 1 && z <= g.nz - 2;
                const bool all_inside = __all_sync(0xFFFFFFFFu, inside || !on);
                if (on) {
                    ++active;
                    if (keys) {
                        on_keys(w, bit, x, y, z, sizeof(T) == 4 && all_inside);
                    } else {
                        const size_t i = flat(g, x, y, z);
                        const uint8_t c = __ldg(a.codes + i);
                        const uint32_t *c0 = a.hp + i;
                        uint32_t t[15];
                        Ext e;
                        if (all_inside) {
#pragma unroll
                            for (int r = 0; r < 15; ++r)
                                t[r] = c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz];
                            e = proxy_ext_interior<true>(t);
                        } else {
                            const uint32_t valid = valid_mask(x, y, z, g.nx, g.ny, g.nz);
#pragma unroll
                            for (int r = 0; r < 15; ++r)
                                t[r] = ((valid >> r) & 1u) ? c0[rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz] : 0u;
                            e = proxy_ext<true>(t);
                        }
                        exact = e.exact;
                        if (exact) outcome(w, bit, x, y, z, e.asc, e.desc, c);
                    }
                }
                const uint32_t md = __ballot_sync(0xFFFFFFFFu, !exact);
                if (md) {
                    if (!exact)
                        sm.defer[warp][ndefer + static_cast<uint32_t>(__popc(md & ((1u << lane) - 1u)))] =
                            make_uint2(static_cast<uint32_t>(w), static_cast<uint32_t>(bit));
                    ndefer += static_cast<uint32_t>(__popc(md));
                    ndeferred += static_cast<uint32_t>(__popc(md));
                    if (ndefer > kSweepDefer - 32) {
                        drain(ndefer - 32, ndefer);
                        ndefer -= 32;
                    }
                }
            });
            drain(0, min(ndefer, 32u));
            if (ndefer > 32) drain(32, ndefer);
            const uint32_t v[8] = {cmax, cmin, cdir, 0u, 0u, 0u, active, 0u};
            block_flush_slot(a.slots + k, v);  // (contains a barrier: sm.deferred is zero before)
            if (sizeof(T) == 4) {
                if (lane == 0 && ndeferred) atomicAdd(&sm.deferred, ndeferred);
                __syncthreads();
                if (threadIdx.x == 0 && sm.deferred) atomicAdd(&a.ls->deferred[k & 1], sm.deferred);
            }
            grid.sync();
            if (sizeof(T) == 4) {
                keys = keys || 10ull * a.ls->deferred[k & 1] > a.slots[k].active;
                if (blockIdx.x == 0 && threadIdx.x == 0) a.ls->deferred[(k + 1) & 1] = 0;
            }
        }
        edits_only = false;
        {
            uint32_t nreq = 0, nchg = 0, nprog = 0;
            for_each_group(sm, a.req, a.freq, g, chunk, [&](bool on, uint32_t w, int bit, int x, int y, int z) {
                uint32_t cb = 0;
                if (on) {
                    const size_t v = flat(g, x, y, z);
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
                        a.hp[v] = proxy_of(nv);
                        cb = 1u << bit;
                    }
                }
                const bool lead = warp_merge_word(on ? w : 0xFFFFFFFFu, cb);
                mark_stencils(nxt, fnxt, g, lead, x >> 5, y, z, cb);
            });
            const uint32_t v[8] = {0u, 0u, 0u, nreq, nchg, nprog, 0u, 0u};
            block_flush_slot(a.slots + k, v);
        }
        grid.sync();
        ++k;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ls->done = k;
}

}  // namespace pmsz
