// naive.cu -- the naive-MSz correction strategy (naive_MSz.cu c_loops,
// 1887-2220): extrema-only sweeps to a fixpoint, then one repair of the
// integral paths whose segmentation labels differ from the original's
// (extract_false_path, naive_MSz.cu:1767-1864), then a check, repeated until
// the check finds no false extremum and no label mismatch.
//
// Layout: the original and current code bytes (steepest ascent rank in the
// low nibble, descent rank in the high nibble; rank 7 = the voxel itself),
// four uint32 label arrays (AS/DS of the original and of the current field),
// one byte per voxel for requests and one for label mismatches, the edit
// counters, and a list of the voxels a pass changed.
//
// The passes change few voxels (a percent at most, mostly some dozens), so what
// bounds them is what is done for all the others, and the launches and waits
// between.  The per-voxel passes read 16 codes, requests or mismatch bytes per
// thread and go on where all are quiet; the codes are brought up to date around
// the changed voxels only; labels are compared as local roots, one hop short of
// finished; extrema sweeps are enqueued a few at a time.  160x144x176 fp64, 32
// passes: 3.7 ms with one voxel per thread, whole-field codes after each pass,
// finished labels and a wait per pass, now 2.0 to 2.2 from run to run; the labels of
// the 14 checks and repairs are half of that.
//
// Semantics per pass are the snapshot ones of the pMSz loop: an extrema sweep
// reads the codes of fhat at its start and applies the union of its requests
// once per voxel, the same outcome as one legal interleaving of the
// reference's in-place kernel; extract_false_path reads only the codes and the
// labels, which it never writes, so its requests are the reference's exactly.
#include "common.cuh"
#include "helpers.cuh"
#include "internal.h"

#include <algorithm>
#include <cstddef>
#include <string>
#include <vector>

namespace pmsz {

namespace {

struct Offsets {
    long long o[15];  // flat offset of every stencil rank
};

Offsets make_offsets(const Geom &g) {
    Offsets t;
    const long long sy = g.nx, sz = static_cast<long long>(g.nx) * g.ny;
    for (int r = 0; r < 15; ++r) t.o[r] = rank_dx(r) + rank_dy(r) * sy + rank_dz(r) * sz;
    return t;
}

inline unsigned grid_for(size_t n) {
    return static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>((n + 255) / 256, 152 * 16)));
}

__device__ __forceinline__ void flush_slot(SweepSlot *slot, uint32_t a, uint32_t b, uint32_t c, uint32_t d,
                                           uint32_t e, uint32_t p, uint32_t act, uint32_t bad) {
    a = warp_sum_u32(a);
    b = warp_sum_u32(b);
    c = warp_sum_u32(c);
    d = warp_sum_u32(d);
    e = warp_sum_u32(e);
    p = warp_sum_u32(p);
    act = warp_sum_u32(act);
    bad = warp_sum_u32(bad);
    if ((threadIdx.x & 31) == 0) {
        if (a) atomicAdd(&slot->fmax, (unsigned long long)a);
        if (b) atomicAdd(&slot->fmin, (unsigned long long)b);
        if (c) atomicAdd(&slot->fdir, (unsigned long long)c);
        if (d) atomicAdd(&slot->requested, (unsigned long long)d);
        if (e) atomicAdd(&slot->changed, (unsigned long long)e);
        if (p) atomicAdd(&slot->progressed, (unsigned long long)p);
        if (act) atomicAdd(&slot->active, (unsigned long long)act);
        if (bad) atomicAdd(&slot->bad, (unsigned long long)bad);
    }
}

// Calls visit(i, o, c) for the voxels whose codes differ (and for a field of
// one voxel, which is both maximum and minimum and never agrees with itself).
// 16 voxels per thread and step: nearly all steps are one comparison.  The
// arrays start at 16-byte boundaries and are padded to them.
template <class Visit>
__device__ __forceinline__ void for_each_differing(const uint8_t *__restrict__ oc, const uint8_t *__restrict__ cc, size_t n,
                                                   Visit &&visit) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x * 16;
    for (size_t i0 = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 16; i0 < n; i0 += stride) {
        const uint4 u = *reinterpret_cast<const uint4 *>(oc + i0), v = *reinterpret_cast<const uint4 *>(cc + i0);
        const uint32_t a[4] = {u.x, u.y, u.z, u.w}, b[4] = {v.x, v.y, v.z, v.w};
        if (((a[0] ^ b[0]) | (a[1] ^ b[1]) | (a[2] ^ b[2]) | (a[3] ^ b[3])) == 0u && n > 1) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (a[k] == b[k] && n > 1) continue;
            for (int j = 0; j < 4; ++j) {
                const size_t i = i0 + 4 * k + j;
                const uint32_t o = (a[k] >> (8 * j)) & 0xFFu, c = (b[k] >> (8 * j)) & 0xFFu;
                if (i < n && (o != c || n == 1)) visit(i, o, c);
            }
        }
    }
}

}  // namespace

// NaN or the 1e30 sentinel in f or fhat (the reference treats 1e30 as a ghost
// cell, pMSz.cu:215): rejected before the loop.
template <typename T>
__global__ void __launch_bounds__(256) k_naive_bad(const T *__restrict__ a, const T *__restrict__ b, size_t n,
                                                   SweepSlot *slot) {
    uint32_t bad = 0;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        bad += (bad_value(a[i]) || bad_value(b[i])) ? 1u : 0u;
    flush_slot(slot, 0, 0, 0, 0, 0, 0, 0, bad);
}

// Extrema-only detection (iscriticle with data_type=0 in naive_MSz.cu:776-826):
// a false or missing maximum requests the voxel itself (false) or its current
// ascent neighbour (missing); a false or missing minimum requests its
// original descent neighbour (false) or the voxel itself (missing).  No
// direction rule.
__global__ void __launch_bounds__(256) k_naive_extrema(const uint8_t *__restrict__ oc, const uint8_t *__restrict__ cc,
                                                       uint8_t *__restrict__ req, size_t n, Offsets off,
                                                       SweepSlot *slot) {
    uint32_t cmax = 0, cmin = 0;
    for_each_differing(oc, cc, n, [&](size_t i, uint32_t o, uint32_t c) {
        const int oa = o & 15, od = o >> 4, ca = c & 15, cd = c >> 4;
        const bool omax = oa == kSelf, omin = !omax && od == kSelf;
        const bool is_max = ca == kSelf, is_min = cd == kSelf;
        if (is_max != omax) {
            ++cmax;
            req[omax ? static_cast<size_t>(static_cast<long long>(i) + off.o[ca]) : i] = 1;
        }
        if (is_min != omin) {
            ++cmin;
            req[omin ? i : static_cast<size_t>(static_cast<long long>(i) + off.o[od])] = 1;
        }
    });
    flush_slot(slot, cmax, cmin, 0, 0, 0, 0, 0, 0);
}

// The integral-path repair (extract_false_path, fix = 0).  For a voxel whose
// DS label differs: follow the original descent while the current descent
// agrees with it and the vertex is not an original extremum; at the stop
// vertex request its original descent neighbour if the current one differs
// (nothing at an original minimum, whose or_types slot is the -2 marker).
// For an AS label mismatch: follow or_types[2c+1] (the original ascent, or the
// original descent at an original maximum) while the current ascent equals
// it; at the stop vertex request its current ascent neighbour if the two
// differ.  Each walk follows a strictly monotone chain of the original order,
// so it ends within n steps; the bound is a guard, counted in `bad` if hit.
// mis: bit 0 where the DS label differs, bit 1 where the AS label does.  A
// block lists the mismatches of its 4096 voxels in shared memory, so that their
// walks are spread over all its threads.
constexpr int kPathSpan = 4096;
__global__ void __launch_bounds__(256) k_naive_paths(const uint8_t *__restrict__ oc, const uint8_t *__restrict__ cc,
                                                     const uint8_t *__restrict__ mis, uint8_t *__restrict__ req, size_t n,
                                                     Offsets off, const unsigned int *open, SweepSlot *slot) {
    if (open && *open) return;  // the mismatches are not settled: the host settles them and comes again
    __shared__ uint16_t s_list[2 * kPathSpan];  // voxel << 1 | kind
    __shared__ uint32_t s_n;
    uint32_t fdir = 0, guard = 0;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const size_t base = static_cast<size_t>(blockIdx.x) * kPathSpan;
    const size_t i0 = base + static_cast<size_t>(threadIdx.x) * 16;
    if (i0 < n) {
        const uint4 u = *reinterpret_cast<const uint4 *>(mis + i0);
        const uint32_t m[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (m[k])
                for (int j = 0; j < 4; ++j) {
                    const uint32_t b = i0 + 4 * k + j < n ? (m[k] >> (8 * j)) & 3u : 0u;
                    if (!b) continue;
                    uint32_t at = atomicAdd(&s_n, static_cast<uint32_t>(__popc(b)));
                    const uint32_t v = threadIdx.x * 16 + 4 * k + j;
                    if (b & 1u) s_list[at++] = static_cast<uint16_t>(v << 1);
                    if (b & 2u) s_list[at] = static_cast<uint16_t>(v << 1 | 1u);
                }
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < s_n; e += blockDim.x) {
        long long cur = static_cast<long long>(base + (s_list[e] >> 1));
        ++fdir;
        bool ok = true;
        if (!(s_list[e] & 1u)) {  // DS
            for (size_t steps = 0;; ++steps) {
                const uint8_t o = oc[cur];
                const int oa = o & 15, od = o >> 4, cd = cc[cur] >> 4;
                const bool omax = oa == kSelf, omin = !omax && od == kSelf;
                if (omax || omin || od != cd) break;
                if (steps >= n) {
                    ok = false;
                    break;
                }
                cur += off.o[od];
            }
            if (ok) {
                const uint8_t o = oc[cur];
                const int oa = o & 15, od = o >> 4, cd = cc[cur] >> 4;
                const bool omin = oa != kSelf && od == kSelf;
                if (!omin && od != cd) req[cur + off.o[od]] = 1;
            } else {
                ++guard;
            }
        } else {  // AS
            bool skip = false;
            for (size_t steps = 0;; ++steps) {
                const uint8_t o = oc[cur];
                const int oa = o & 15, od = o >> 4, ca = cc[cur] & 15;
                const int r1 = oa == kSelf ? od : oa;
                if (r1 != ca) break;
                if (r1 == kSelf) {  // a vertex that is its own successor in both fields
                    skip = true;
                    break;
                }
                if (steps >= n) {
                    ok = false;
                    break;
                }
                cur += off.o[r1];
            }
            if (!ok) {
                ++guard;
            } else if (!skip) {
                const uint8_t o = oc[cur];
                const int oa = o & 15, od = o >> 4, ca = cc[cur] & 15;
                const int r1 = oa == kSelf ? od : oa;
                if (r1 != ca) req[cur + off.o[ca]] = 1;
            }
        }
    }
    flush_slot(slot, 0, 0, fdir, 0, 0, 0, 0, guard);
}

// The edits of one pass: every requested voxel once (applyDeltaBuffer_local,
// naive_MSz.cu:620-641), the request cleared; the voxels whose value changed
// go to list (the first `cap` of them; *listed counts all).
template <typename T>
__global__ void __launch_bounds__(256) k_naive_apply(const T *__restrict__ f, T *__restrict__ fh,
                                                     uint8_t *__restrict__ cnt, uint8_t *__restrict__ req, size_t n,
                                                     T eps, T delta, int q, uint32_t *__restrict__ list, uint32_t cap,
                                                     uint32_t *listed, SweepSlot *slot) {
    uint32_t rq = 0, ch = 0, pr = 0;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x * 16;
    for (size_t i0 = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 16; i0 < n; i0 += stride) {
        const uint4 u = *reinterpret_cast<const uint4 *>(req + i0);
        if (!(u.x | u.y | u.z | u.w)) continue;
        *reinterpret_cast<uint4 *>(req + i0) = make_uint4(0u, 0u, 0u, 0u);
        const uint32_t m[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            for (uint32_t b = m[k] & 0x01010101u; b; b &= b - 1) {
                const size_t i = i0 + 4 * k + static_cast<size_t>((__ffs(b) - 1) >> 3);
                bool progressed = false;
                if (apply_one(f, fh, cnt, i, eps, delta, q, progressed)) {
                    ++ch;
                    // one atomic for the lanes that are here together
                    const uint32_t here = __activemask(), lane = threadIdx.x & 31u, lead = __ffs(here) - 1u;
                    uint32_t at = lane == lead ? atomicAdd(listed, static_cast<uint32_t>(__popc(here))) : 0u;
                    at = __shfl_sync(here, at, static_cast<int>(lead)) + static_cast<uint32_t>(__popc(here & ((1u << lane) - 1u)));
                    if (at < cap) list[at] = static_cast<uint32_t>(i);
                }
                pr += progressed ? 1u : 0u;
                ++rq;
            }
    }
    flush_slot(slot, 0, 0, 0, rq, ch, pr, 0, 0);
}

// The codes of fh around the changed voxels: of every voxel whose stencil holds
// one (16 threads per changed voxel; a voxel reached twice gets the same byte
// twice).  Where the list overflowed, of all voxels.
template <typename T>
__global__ void __launch_bounds__(256) k_naive_recode(const T *__restrict__ fh, const uint32_t *__restrict__ list,
                                                      const uint32_t *listed, uint32_t cap, uint8_t *__restrict__ codes,
                                                      Geom g) {
    const uint32_t m = *listed;
    const bool all = m > cap;
    const size_t total = all ? g.n : static_cast<size_t>(m) * 16;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += stride) {
        const int r = static_cast<int>(e & 15u);
        if (!all && r == 15) continue;
        const uint32_t v = all ? static_cast<uint32_t>(e) : list[e >> 4];
        const uint32_t row = fdiv(v, g.div_nx), zz = fdiv(row, g.div_ny);
        int x = static_cast<int>(v - row * static_cast<uint32_t>(g.nx)), y = static_cast<int>(row - zz * static_cast<uint32_t>(g.ny)),
            z = static_cast<int>(zz);
        if (!all) {  // the stencil is symmetric: its points are also the voxels it belongs to
            if (!((valid_mask(x, y, z, g.nx, g.ny, g.nz) >> r) & 1u)) continue;
            x += rank_dx(r);
            y += rank_dy(r);
            z += rank_dz(r);
        }
        const size_t i = flat(g, x, y, z);
        const uint32_t valid = valid_mask(x, y, z, g.nx, g.ny, g.nz);
        typename KeyOf<T>::type k[15];
        load_keys(fh, i, g, valid, k);
        int asc, desc;
        arg_ext(k, valid, asc, desc);
        codes[i] = static_cast<uint8_t>(asc | (desc << 4));
    }
}

// The label mismatches of the current field (mis, as k_naive_paths reads them),
// as0 / ds0 finished, as1 / ds1 one hop short of it (hop) or finished.  With a
// slot, the check (iscriticle with checkFinal = 1, then extract_false_path with
// fix = 1): false/missing extrema, and per voxel one count for a DS label
// mismatch, else one for an AS label mismatch.  Four voxels per thread and step.
__global__ void __launch_bounds__(256) k_naive_compare(const uint8_t *__restrict__ oc, const uint8_t *__restrict__ cc,
                                                       const uint32_t *__restrict__ as0, const uint32_t *__restrict__ ds0,
                                                       const uint32_t *__restrict__ as1, const uint32_t *__restrict__ ds1,
                                                       int hop, size_t n, uint8_t *__restrict__ mis, SweepSlot *slot) {
    uint32_t cmax = 0, cmin = 0, cdir = 0;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x * 4;
    for (size_t i0 = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 4; i0 < n; i0 += stride) {
        const uint4 a0 = *reinterpret_cast<const uint4 *>(as0 + i0), d0 = *reinterpret_cast<const uint4 *>(ds0 + i0);
        const uint4 a1 = *reinterpret_cast<const uint4 *>(as1 + i0), d1 = *reinterpret_cast<const uint4 *>(ds1 + i0);
        const uint32_t o4 = *reinterpret_cast<const uint32_t *>(oc + i0), c4 = *reinterpret_cast<const uint32_t *>(cc + i0);
        const uint32_t A0[4] = {a0.x, a0.y, a0.z, a0.w}, D0[4] = {d0.x, d0.y, d0.z, d0.w};
        uint32_t A1[4] = {a1.x, a1.y, a1.z, a1.w}, D1[4] = {d1.x, d1.y, d1.z, d1.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (hop && i0 + j < n) {
                A1[j] = as1[A1[j]];
                D1[j] = ds1[D1[j]];
            }
        uint32_t m4 = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t m = i0 + j < n ? (D0[j] != D1[j] ? 1u : 0u) | (A0[j] != A1[j] ? 2u : 0u) : 0u;
            m4 |= m << (8 * j);
            cdir += m != 0;
        }
        *reinterpret_cast<uint32_t *>(mis + i0) = m4;
        if (slot && (o4 != c4 || n == 1)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t o = (o4 >> (8 * j)) & 0xFFu, c = (c4 >> (8 * j)) & 0xFFu;
                const int oa = o & 15, od = o >> 4, ca = c & 15, cd = c >> 4;
                const bool omax = oa == kSelf, omin = !omax && od == kSelf;
                if (i0 + j < n) {
                    cmax += (ca == kSelf) != omax;
                    cmin += (cd == kSelf) != omin;
                }
            }
        }
    }
    if (slot) flush_slot(slot, cmax, cmin, cdir, 0, 0, 0, 0, 0);
}

// What the host reads back together.
constexpr int kNaiveAhead = 4;  // extrema sweeps enqueued at a time
struct NaiveState {
    SweepSlot slot[kNaiveAhead];
    uint32_t listed[kNaiveAhead];  // voxels changed by the pass (k_naive_recode reads it)
    // labels_roots' words: of the original, the current field before the repair, and after it
    unsigned int open0[2], open1[2], open2[2];
};

template <typename T>
int naive_impl(const T *f, T *fh, size_t nx, size_t ny, size_t nz, double eb, const pmsz_opts *opts,
               pmsz_result *res, cudaStream_t s) {
    if (!f || !fh) return set_error(PMSZ_ERR_ARG, "null field pointer");
    int rc = check_geom(nx, ny, nz);
    if (rc) return rc;
    const int q = opts ? opts->q : 5;
    const int64_t max_sweeps = opts ? opts->max_sweeps : 10000;
    if (!(eb > 0.0) || q < 1 || q > 255 || max_sweeps < 1)
        return set_error(PMSZ_ERR_ARG, "need eb > 0, 1 <= q <= 255 and max_sweeps >= 1");
    const Geom g = make_geom(nx, ny, nz);
    if (g.n >= (static_cast<size_t>(1) << 32))
        return set_error(PMSZ_ERR_ARG, "the naive strategy's labels need fewer than 2^32 voxels");
    const size_t n = g.n;
    const T eps = static_cast<T>(eb), delta = static_cast<T>(eb / q);
    const Offsets off = make_offsets(g);
    const unsigned grid = grid_for(n), grid16 = grid_for((n + 15) / 16), grid4 = grid_for((n + 3) / 4);
    // changed voxels a pass may list: beyond a 32nd of the field, recoding all
    // voxels costs less than the 15 around each
    const uint32_t cap = static_cast<uint32_t>(std::max<size_t>(n / 32, 64));

    Workspace ws(s);
    const size_t o_oc = ws.reserve<uint8_t>(n), o_cc = ws.reserve<uint8_t>(n), o_cnt = ws.reserve<uint8_t>(n),
                 o_req = ws.reserve<uint8_t>(n), o_mis = ws.reserve<uint8_t>(n);
    const size_t o_as0 = ws.reserve<uint32_t>(n), o_ds0 = ws.reserve<uint32_t>(n), o_as1 = ws.reserve<uint32_t>(n),
                 o_ds1 = ws.reserve<uint32_t>(n);
    const size_t o_state = ws.reserve<NaiveState>(1), o_list = ws.reserve<uint32_t>(cap);
    const size_t o_exits = ws.reserve<uint32_t>(label_list_words(nx, ny, nz));
    if ((rc = ws.commit())) return rc;
    uint8_t *oc = ws.at<uint8_t>(o_oc), *cc = ws.at<uint8_t>(o_cc), *cnt = ws.at<uint8_t>(o_cnt),
            *req = ws.at<uint8_t>(o_req), *mis = ws.at<uint8_t>(o_mis);
    uint32_t *as0 = ws.at<uint32_t>(o_as0), *ds0 = ws.at<uint32_t>(o_ds0), *as1 = ws.at<uint32_t>(o_as1),
             *ds1 = ws.at<uint32_t>(o_ds1), *list = ws.at<uint32_t>(o_list), *exits = ws.at<uint32_t>(o_exits);
    NaiveState *st = ws.at<NaiveState>(o_state);
    NaiveState *hs = static_cast<NaiveState *>(host_pinned(sizeof(NaiveState)));
    if (!hs) return set_error(PMSZ_ERR_OOM, "pinned host allocation failed");
    NaiveState got;  // (the jumping of labels_complete reads back through the same pinned block)

    EventTimer et;
    if ((rc = et.init())) return rc;
    PMSZ_CUDA(cudaEventRecord(et.ev[0], s));
    int64_t launches = 0;
    auto read_state = [&]() -> int {
        PMSZ_CUDA(cudaMemcpyAsync(hs, st, sizeof(NaiveState), cudaMemcpyDeviceToHost, s));
        PMSZ_CUDA(cudaStreamSynchronize(s));
        got = *hs;
        return PMSZ_OK;
    };
    auto clear_passes = [&]() -> int {  // the slots and the lists' lengths
        PMSZ_CUDA(cudaMemsetAsync(st, 0, offsetof(NaiveState, open0), s));
        return PMSZ_OK;
    };

    PMSZ_CUDA(cudaMemsetAsync(cnt, 0, n, s));
    PMSZ_CUDA(cudaMemsetAsync(req, 0, (n + 15) / 16 * 16, s));  // (read 16 at a time)
    PMSZ_CUDA(cudaMemsetAsync(st, 0, sizeof(NaiveState), s));
    k_naive_bad<T><<<grid, 256, 0, s>>>(f, fh, n, st->slot);
    PMSZ_CUDA(cudaGetLastError());
    ++launches;
    if ((rc = read_state())) return rc;
    if (got.slot[0].bad) return set_error(PMSZ_ERR_ARG, "input holds NaN or the 1e30 ghost sentinel");

    // original codes and labels (iscriticle data_type=1 + PathCompression,
    // naive_MSz.cu:1910-1917)
    if ((rc = codes_impl<T>(f, nx, ny, nz, oc, s))) return rc;
    if ((rc = labels_roots(oc, nx, ny, nz, as0, ds0, exits, st->open0, s))) return rc;
    if ((rc = labels_finish(nx, ny, nz, as0, ds0, s))) return rc;
    bool original_checked = false;
    // after a read_state: the original's labels in full, once
    auto settle_original = [&]() -> int {
        if (original_checked) return PMSZ_OK;
        original_checked = true;
        return got.open0[0] ? labels_complete(nx, ny, nz, as0, ds0, st->open0, s) : PMSZ_OK;
    };

    std::vector<SweepSlot> log;
    int status = PMSZ_ERR_NOT_CONVERGED;
    std::string why = "max_sweeps reached";
    uint64_t hmax = 1, hmin = 1, edits = 0;
    int64_t outer = 0, inner = 0;
    bool codes_current = false;   // cc describes the current fhat
    bool labels_current = false;  // and mis its labels
    auto record = [&](const SweepSlot &r) { log.push_back(r); };
    auto room = [&]() { return max_sweeps - static_cast<int64_t>(log.size()); };
    // the edits of pass p, and the codes they leave
    auto apply_pass = [&](int p) -> int {
        k_naive_apply<T><<<grid16, 256, 0, s>>>(f, fh, cnt, req, n, eps, delta, q, list, cap, &st->listed[p], &st->slot[p]);
        k_naive_recode<T><<<152 * 4, 256, 0, s>>>(fh, list, &st->listed[p], cap, cc, g);
        PMSZ_CUDA(cudaGetLastError());
        launches += 2;
        return PMSZ_OK;
    };
    // label mismatches of the current codes into mis; with a slot, the check
    auto compare = [&](int hop, SweepSlot *slot) -> int {
        k_naive_compare<<<grid4, 256, 0, s>>>(oc, cc, as0, ds0, as1, ds1, hop, n, mis, slot);
        PMSZ_CUDA(cudaGetLastError());
        ++launches;
        return PMSZ_OK;
    };

    for (;;) {
        ++outer;
        uint64_t progressed_outer = 0;
        bool stuck = false;
        while (hmax || hmin) {  // extrema-only sweeps
            if (room() <= 0) goto done;
            if (!codes_current && (rc = codes_impl<T>(fh, nx, ny, nz, cc, s))) return rc;
            codes_current = true;
            // A few sweeps at once: one that follows the end of the loop below
            // requests nothing (no false extremum), or the same voxels that it
            // could not change, and so changes nothing either.
            const int ahead = static_cast<int>(std::min<int64_t>(kNaiveAhead, room()));
            if ((rc = clear_passes())) return rc;
            for (int p = 0; p < ahead; ++p) {
                k_naive_extrema<<<grid16, 256, 0, s>>>(oc, cc, req, n, off, &st->slot[p]);
                PMSZ_CUDA(cudaGetLastError());
                ++launches;
                if ((rc = apply_pass(p))) return rc;
            }
            if ((rc = read_state()) || (rc = settle_original())) return rc;
            labels_current = false;
            for (int p = 0; p < ahead && (hmax || hmin); ++p) {
                const SweepSlot &r = got.slot[p];
                ++inner;
                record(r);
                edits += r.requested;
                progressed_outer += r.progressed;
                hmax = r.fmax;
                hmin = r.fmin;
                if ((hmax || hmin) && r.progressed == 0) {
                    stuck = true;
                    break;
                }
            }
            if (stuck) break;
        }
        if (stuck) {
            why = "a sweep changed nothing";
            goto done;
        }
        // path repair, and the check behind it where the log has room for both
        if (room() <= 0) goto done;
        const unsigned int *open = nullptr;
        if (!labels_current) {
            if ((rc = labels_roots(cc, nx, ny, nz, as1, ds1, exits, st->open1, s)) || (rc = compare(1, nullptr))) return rc;
            open = st->open1;
        }
        const bool both = room() >= 2;
        for (;;) {
            if ((rc = clear_passes())) return rc;
            k_naive_paths<<<static_cast<unsigned>((n + kPathSpan - 1) / kPathSpan), 256, 0, s>>>(oc, cc, mis, req, n, off, open,
                                                                                                 &st->slot[0]);
            PMSZ_CUDA(cudaGetLastError());
            ++launches;
            if ((rc = apply_pass(0))) return rc;
            if (both && ((rc = labels_roots(cc, nx, ny, nz, as1, ds1, exits, st->open2, s)) || (rc = compare(1, &st->slot[1]))))
                return rc;
            if ((rc = read_state())) return rc;
            if (!open || !got.open1[0]) break;
            // chains beyond the walks' bounds, and so no pass yet: the labels in full first
            if (!both && (rc = labels_roots(cc, nx, ny, nz, as1, ds1, exits, st->open1, s))) return rc;
            if ((rc = labels_complete(nx, ny, nz, as1, ds1, st->open1, s)) || (rc = compare(0, nullptr))) return rc;
            open = nullptr;
        }
        if (got.slot[0].bad) {
            status = PMSZ_ERR_CUDA;
            why = "an integral-path walk exceeded its bound";
            goto done;
        }
        record(got.slot[0]);
        edits += got.slot[0].requested;
        progressed_outer += got.slot[0].progressed;
        if (!both) goto done;
        if (got.open2[0]) {  // chains beyond the walks' bounds: the labels in full, and the check once more
            if ((rc = labels_complete(nx, ny, nz, as1, ds1, st->open2, s)) || (rc = clear_passes()) ||
                (rc = compare(0, &st->slot[1])) || (rc = read_state()))
                return rc;
        }
        labels_current = true;
        const SweepSlot &r = got.slot[1];
        record(r);
        if (!r.fmax && !r.fmin && !r.fdir) {
            status = PMSZ_OK;
            goto done;
        }
        if (!progressed_outer) {
            why = "an outer iteration changed nothing";
            goto done;
        }
        hmax = r.fmax;
        hmin = r.fmin;
    }
done:
    PMSZ_CUDA(cudaEventRecord(et.ev[1], s));
    PMSZ_CUDA(cudaEventSynchronize(et.ev[1]));
    float ms_total = 0;
    PMSZ_CUDA(cudaEventElapsedTime(&ms_total, et.ev[0], et.ev[1]));
    if (res) {
        res->sweeps = static_cast<int64_t>(log.size());
        res->iteration = 2 * outer + inner;
        res->edits = edits;
        if (res->sweep_log)
            for (int64_t k = 0; k < std::min<int64_t>(res->sweeps, res->sweep_log_cap); ++k) {
                const SweepSlot &r = log[static_cast<size_t>(k)];
                res->sweep_log[k] = pmsz_sweep_record{r.fmax, r.fmin, r.fdir, r.requested,
                                                      r.changed, r.progressed, r.active, r.bad};
            }
        res->ms_first_pass = res->ms_detect = res->ms_apply = 0.0;
        res->launches = launches;
        res->ms_total = ms_total;
    }
    if ((rc = ws.release())) return rc;
    if (status == PMSZ_ERR_NOT_CONVERGED) return set_error(status, "naive strategy did not converge: " + why);
    if (status != PMSZ_OK) return set_error(status, why);
    return PMSZ_OK;
}

template int naive_impl<float>(const float *, float *, size_t, size_t, size_t, double, const pmsz_opts *,
                               pmsz_result *, cudaStream_t);
template int naive_impl<double>(const double *, double *, size_t, size_t, size_t, double, const pmsz_opts *,
                                pmsz_result *, cudaStream_t);

}  // namespace pmsz

using namespace pmsz;

extern "C" int pmsz_correct_naive_f32(const float *f, float *fhat, size_t nx, size_t ny, size_t nz, double eb,
                                      const pmsz_opts *opts, pmsz_result *res, void *stream) {
    return guarded([&] { return naive_impl<float>(f, fhat, nx, ny, nz, eb, opts, res, as_stream(stream)); });
}
extern "C" int pmsz_correct_naive_f64(const double *f, double *fhat, size_t nx, size_t ny, size_t nz, double eb,
                                      const pmsz_opts *opts, pmsz_result *res, void *stream) {
    return guarded([&] { return naive_impl<double>(f, fhat, nx, ny, nz, eb, opts, res, as_stream(stream)); });
}
