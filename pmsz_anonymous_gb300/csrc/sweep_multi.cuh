// sweep_multi.cuh -- the sweeps of many fields in one cooperative launch, the
// form of k_sweeps (sweep.cuh) for pmsz_correct_batch and the server; included
// by batch.cu.
//
// Two tables of fields, fp32 and fp64, step through their sweeps together:
// one grid barrier after the detection of all of them and one after their
// edits, so small fields of either type fill the chip side by side.  Every
// block applies each field's stop rule to the field's last slot; a field that
// has stopped is skipped from then on.
//
// The groups of a table's fields lie end to end, each field's count rounded up
// to whole chunks of eight groups, and the chunks are dealt to the warps as in
// k_sweeps; the field of a thread's first chunk is looked up once per launch.
// The up to four groups that a warp visits at a time are of one field, so its
// pointers and strides are the same for the whole warp, and its counters stay
// in registers until the warp's next field (a block's list is in field order:
// once per field and phase at most).
//
// Measured: 32 fp32 fields (116 million voxels) 8.7 -> 5.1 ms end to end, from
// compacted lists in a conditional CUDA graph and a cooperative tail (4.9 ms of
// kernels, and the gaps between them) to one launch of 3.4 ms; a burst of 24
// mixed jobs through the server 8.6 -> 3.6 ms.
#pragma once
#include "batch.h"
#include "sweep.cuh"

namespace pmsz {

// Largest i with pre[i] <= r; empty segments (pre[i] == pre[i + 1]) are never
// the answer for an r below pre[n].
__device__ __forceinline__ int find_seg(const uint32_t *__restrict__ pre, int n, uint32_t r) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(pre + mid) <= r) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

struct FieldMasks {
    uint32_t edits[kMaxBatch / 32];   // fields that run this iteration
    uint32_t detect[kMaxBatch / 32];  // of those, not in their first
};
struct MultiSmem {
    SweepSmem s;
    uint32_t local[kSweepBlock];  // the field's group at each thread's chunk,
    uint16_t field[kSweepBlock];  // and the field
    FieldMasks m32, m64;
    // the table row of each warp's field (from here its pointers are reloaded
    // at will; a row in global memory would be after every store)
    alignas(16) unsigned char row[kSweepWarps][sizeof(Inst<double>)];
    SweepStep step[kSweepWarps][15];  // its request steps
};
static_assert(sizeof(Inst<float>) <= sizeof(Inst<double>) && sizeof(Inst<float>) % 8 == 0 && sizeof(Inst<double>) % 8 == 0,
              "rows are copied by words");

__device__ __forceinline__ bool mask_bit(const uint32_t *m, int i) { return (m[i >> 5] >> (i & 31)) & 1u; }

template <typename T>
__device__ __forceinline__ SweepSlot *slot_of(const Inst<T> &I, int64_t k) {
    return I.slots + k * I.stride;
}

// Adds a warp's counters (v[c] to 64-bit counter first + c, c < 4) to a slot.
__device__ __forceinline__ void warp_flush_slot(SweepSlot *slot, int first, uint32_t (&v)[4]) {
    const int lane = threadIdx.x & 31;
    uint32_t mine = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t t = warp_sum_u32(v[c]);
        if (lane == c) mine = t;
        v[c] = 0;
    }
    if (mine) atomicAdd(reinterpret_cast<unsigned long long *>(slot) + first + lane, static_cast<unsigned long long>(mine));
}

// The masks of iteration `it`; returns whether this thread's warp saw a field
// run, and in `stopped` whether it saw one stop.
template <typename T>
__device__ __forceinline__ bool field_masks(FieldMasks &m, const SweepTable<T> &t, int64_t it, bool &stopped) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t any = 0, stop = 0;
    for (int w = warp; w < (t.n + 31) / 32; w += kSweepWarps) {
        const int i = w * 32 + lane;
        const bool was = it == 0 ? i < t.n && t.inst[i].active : mask_bit(m.edits, i);
        bool run = was, fresh = false;
        if (was) {
            const Inst<T> &I = t.inst[i];
            const int64_t s = I.k + it;
            fresh = it == 0 && I.first;
            if (!fresh) {
                const SweepSlot *p = slot_of(I, s - 1);
                run = !sweep_stops(p->fmax, p->fmin, p->fdir, p->progressed, s, I.max_sweeps) && !(s == 1 && p->bad);
            }
        }
        const uint32_t e = __ballot_sync(0xFFFFFFFFu, run), d = __ballot_sync(0xFFFFFFFFu, run && !fresh), b = __ballot_sync(0xFFFFFFFFu, was);
        if (lane == 0) {
            m.edits[w] = e;
            m.detect[w] = d;
        }
        any |= e;
        stop |= b & ~e;
    }
    stopped = stop != 0;
    return any != 0;
}

// One phase (0: detection, 1: edits) of iteration `it` over a table.  home,
// home_local: the field and the field's group of this thread's first chunk.
template <typename T, int PHASE>
__device__ __forceinline__ void multi_phase(MultiSmem &ms, const FieldMasks &m, const SweepTable<T> &t, uint32_t chunk,
                                            int64_t it, int home, uint32_t home_local) {
    SweepSmem &sm = ms.s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t *mask = PHASE == 0 ? m.detect : m.edits;
    const uint64_t nc = static_cast<uint64_t>(t.chunks) * (8u / chunk);
    int cf = -1;  // the field whose counters are in v
    uint32_t v[4] = {0u, 0u, 0u, 0u}, ndefer = 0;

    const Inst<T> &I = *reinterpret_cast<const Inst<T> *>(ms.row[warp]);  // of field cf

    auto leave = [&] {  // the warp is done with field cf
        const int64_t s = I.k + it;
        if (PHASE == 0) {
            SweepSlot *slot = slot_of(I, s);
            if (lane == 0 && v[3]) atomicAdd(&slot->active, static_cast<unsigned long long>(v[3]));
            v[3] = 0;
            warp_flush_slot(slot, 0, v);
        } else {
            warp_flush_slot(slot_of(I, s), 3, v);
        }
    };

    for (uint64_t base = 0; base < nc; base += static_cast<uint64_t>(kSweepBlock) * gridDim.x) {
        const uint64_t c = base + static_cast<uint64_t>(threadIdx.x) * gridDim.x + blockIdx.x;
        uint32_t fm = 0, local = home_local;
        int fi = home;
        if (c < nc) {
            if (base) {
                const uint32_t c8 = static_cast<uint32_t>(c * chunk / 8);
                fi = find_seg(t.cpre, t.n, c8);
                local = static_cast<uint32_t>(c * chunk - static_cast<uint64_t>(__ldg(t.cpre + fi)) * 8u);
            }
            if (mask_bit(mask, fi)) {
                const Inst<T> &J = t.inst[fi];
                uint8_t *flag = (PHASE == 1 ? J.freq : ((J.k + it) & 1) ? J.f1 : J.f0) + local;
                fm = chunk_flags(flag, chunk);  // (padded to whole chunks of eight)
                if (fm) clear_chunk_flags(flag, chunk);
            }
        }
        const uint32_t cnt = static_cast<uint32_t>(__popc(fm));
        uint32_t inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) sm.groups[warp] = inc;
        if (threadIdx.x == 0) sm.next = 0;
        ms.local[threadIdx.x] = local;
        ms.field[threadIdx.x] = static_cast<uint16_t>(fi);
        __syncthreads();
        uint32_t first = inc - cnt, groups = 0;
#pragma unroll
        for (int k = 0; k < kSweepWarps; ++k) {
            const uint32_t n = sm.groups[k];
            first += k < warp ? n : 0u;
            groups += n;
        }
        for (; fm; fm &= fm - 1, ++first) sm.group[first] = static_cast<uint16_t>(threadIdx.x * 8 + __ffs(fm) - 1);
        __syncthreads();
        const uint32_t rounds = (groups + 4 * kSweepWarps - 1) / (4 * kSweepWarps);
        const uint32_t share = groups ? (groups + kSweepWarps * rounds - 1) / (kSweepWarps * rounds) : 1u;
        // the next up to `share` groups that are of one field: the field (-1:
        // none left), this lane's word and its index
        uint32_t at = 0, end = 0;
        auto take = [&](int &f, uint64_t &w) -> uint32_t {
            if (at >= end) {
                at = lane == 0 ? atomicAdd(&sm.next, share) : 0u;
                at = __shfl_sync(0xFFFFFFFFu, at, 0);
                end = min(at + share, groups);
            }
            f = -1;
            w = ~0ull;
            if (at >= end) return 0u;
            f = ms.field[sm.group[at] >> 3];
            const bool same = lane < 4 && at + lane < end && ms.field[sm.group[at + lane] >> 3] == f;
            const uint32_t run = static_cast<uint32_t>(__popc(__ballot_sync(0xFFFFFFFFu, same)));
            const Inst<T> &J = t.inst[f];
            const uint32_t *bm = PHASE == 1 ? J.req : ((J.k + it) & 1) ? J.act1 : J.act0;
            if (static_cast<uint32_t>(lane >> 3) < run) {
                const uint32_t e = sm.group[at + (lane >> 3)];
                w = static_cast<uint64_t>(ms.local[e >> 3] + (e & 7u)) * kGroupWords + (lane & 7);
            }
            at += run;
            return w < J.g.nwords ? bm[w] : 0u;
        };
        int f, f_next;
        uint64_t w, w_next;
        uint32_t word = take(f, w);
        for (; f >= 0; f = f_next, w = w_next) {
            const uint32_t next = take(f_next, w_next);  // in flight while these groups are visited
            if (f != cf) {
                if (cf >= 0) leave();
                cf = f;
                __syncwarp();
                for (uint32_t b = lane; b < sizeof(Inst<T>) / 4; b += 32)
                    reinterpret_cast<uint32_t *>(ms.row[warp])[b] = __ldg(reinterpret_cast<const uint32_t *>(t.inst + f) + b);
                __syncwarp();
                fill_steps(ms.step[warp], I.g, lane);
                __syncwarp();
            }
            const Geom &g = I.g;
            const bool odd = ((I.k + it) & 1) != 0;
            uint32_t *nxt = odd ? I.act0 : I.act1;
            uint8_t *fnxt = odd ? I.f0 : I.f1;
            if (word) (PHASE == 1 ? I.req : odd ? I.act1 : I.act0)[w] = 0;
            const uint32_t total = list_words(sm, g, w, word);
            if (PHASE == 0)
                detect_words<T>(sm, I, ms.step[warp], nxt, fnxt, total, static_cast<uint32_t>(w),
                                f_next != f, v, ndefer);
            else
                edit_words<T>(sm, I, nxt, fnxt, total, v);
            __syncwarp();  // list and at are rewritten by the next groups
            word = next;
        }
        __syncthreads();  // the lists are rewritten by the next chunks, or by the other table
    }
    if (cf >= 0) leave();
}

// The field and group of this thread's first chunk of a table.
template <typename T>
__device__ __forceinline__ void first_chunk(const SweepTable<T> &t, uint32_t chunk, int &fi, uint32_t &local) {
    const uint64_t c = static_cast<uint64_t>(threadIdx.x) * gridDim.x + blockIdx.x;
    fi = 0;
    local = 0;
    if (c < static_cast<uint64_t>(t.chunks) * (8u / chunk)) {
        fi = find_seg(t.cpre, t.n, static_cast<uint32_t>(c * chunk / 8));
        local = static_cast<uint32_t>(c * chunk - static_cast<uint64_t>(__ldg(t.cpre + fi)) * 8u);
    }
}

// What the server reads of each field once the launch has ended.
template <typename T>
__device__ __forceinline__ void write_reports(const FieldMasks &m, const SweepTable<T> &t, int64_t it) {
    for (int i = threadIdx.x; t.report && i < t.n; i += kSweepBlock) {
        const Inst<T> &I = t.inst[i];
        if (!I.active) continue;
        SweepReport r{};
        r.sweeps = I.k + it;
        r.running = mask_bit(m.edits, i) ? 1 : 0;
        if (!r.running && r.sweeps > 0) {
            r.last = *slot_of(I, r.sweeps - 1);
            for (int64_t s = 0; s < r.sweeps; ++s) r.edits += slot_of(I, s)->requested;
        }
        t.report[i] = r;
    }
}

// Bound like k_sweeps by gather latency and, for small sets, by the barriers
// (about 2 us each).  Ends when no field runs, when a field stops and
// a.until_stop is set, or when the host has set *a.yield (polled once a sweep;
// every block sees the same value, through ctl->yield).
__global__ void __launch_bounds__(kSweepBlock, 3) k_sweeps_multi(const __grid_constant__ MultiSweeps a) {
    __shared__ MultiSmem ms;
    uint32_t target = 0;  // of the grid barrier
    const bool first = blockIdx.x == 0;
    auto chunk_for = [&](uint64_t chunks) -> uint32_t {  // as in k_sweeps
        uint32_t c = 8;
        while (c > 1 && chunks * 8u < static_cast<uint64_t>(c) * gridDim.x * kSweepWarps) c >>= 1;
        return c;
    };
    const uint32_t c32 = chunk_for(a.t32.chunks), c64 = chunk_for(a.t64.chunks);
    int home32, home64;
    uint32_t local32, local64;
    first_chunk(a.t32, c32, home32, local32);
    first_chunk(a.t64, c64, home64, local64);
    clear_bits(ms.s.bits[threadIdx.x >> 5]);
    int64_t it = 0;
    while (true) {
        bool stop32 = false, stop64 = false;
        const bool run = field_masks(ms.m32, a.t32, it, stop32) | field_masks(ms.m64, a.t64, it, stop64);
        const bool yield = it > 0 && a.yield && a.ctl->yield[(it - 1) & 1];
        const int more = __syncthreads_or(run);
        const int stopped = __syncthreads_or(stop32 || stop64);
        if (!more || (a.until_stop && stopped) || yield) break;
        int want = 0;
        if (a.yield && first && threadIdx.x == 0) want = *a.yield;  // read while the sweep runs
        multi_phase<float, 0>(ms, ms.m32, a.t32, c32, it, home32, local32);
        multi_phase<double, 0>(ms, ms.m64, a.t64, c64, it, home64, local64);
        if (!sweep_barrier(&a.ctl->bar, target, &a.ctl->err)) return;
        multi_phase<float, 1>(ms, ms.m32, a.t32, c32, it, home32, local32);
        multi_phase<double, 1>(ms, ms.m64, a.t64, c64, it, home64, local64);
        if (a.yield && first && threadIdx.x == 0) a.ctl->yield[it & 1] = want;
        if (!sweep_barrier(&a.ctl->bar, target, &a.ctl->err)) return;
        ++it;
    }
    if (first) {
        write_reports(ms.m32, a.t32, it);
        write_reports(ms.m64, a.t64, it);
        if (threadIdx.x == 0) a.ctl->iters = it;
    }
}

}  // namespace pmsz
