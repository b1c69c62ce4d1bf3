// correct.cu -- labelling, detection and edit kernels and the correction loop.
//
// Replaces iscriticle (pMSz.cu:649-899), applyDeltaBuffer_local
// (pMSz.cu:623-645), init_edits / init_counter (pMSz.cu:902-906, 1745-1749) and
// the host loop c_loops (pMSz.cu:1872-2074) at an MPI grid of 1x1x1.
//
// Sweep k (snapshot semantics):
//   detect   every voxel u of the active set A_k reads fhat on its closed
//            stencil N[u] and the original direction code of u, applies the
//            reference rules, ORs the vertices it wants lowered into the
//            request bitmap R, and sets u in M_k (the next active bitmap) if
//            it mismatched.
//   apply    every vertex in R is edited once (applyDeltaBuffer_local); R is
//            cleared; the closed stencil of every vertex whose value changed
//            is ORed into the next active bitmap.
// A voxel whose stencil did not change keeps its previous outcome, so
// A_{k+1} = M_k U N[C_k] (C_k = changed vertices) yields exactly the requests
// and counters of a full sweep over all voxels.  Sweep 1 is a full pass fused
// with the original labelling: it reads f and fhat once and writes the codes.
// PMSZ_FLAG_FULL_SWEEPS replaces the active set by the whole field.
#include "common.cuh"
#include "../../include/pmsz.h"
#include "helpers.cuh"
#include "internal.h"

#include <cudaTypedefs.h>  // PFN_cuTensorMapEncodeTiled

#include <algorithm>
#include <cstring>
#include <chrono>
#include <iterator>
#include <mutex>
#include <string>
#include <tuple>
#include <utility>
#include <vector>

namespace pmsz {

// ---------------------------------------------------------------------------
// Full detection pass over a 3-D grid: block (32, 8), one warp per 32-voxel
// x-segment, which is exactly one bitmap word.  FIRST: also label the
// original field f and store the code byte (iscriticle data_type=1 fused with
// the first data_type=0 pass).
// ---------------------------------------------------------------------------
template <typename T, bool FIRST>
__global__ void __launch_bounds__(256) k_detect_full(const T *__restrict__ f, const T *__restrict__ fh,
                                                     uint8_t *__restrict__ codes, uint32_t *__restrict__ req,
                                                     uint32_t *__restrict__ act_next, SweepSlot *slot, Geom g) {
    using K = typename KeyOf<T>::type;
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z;
    const bool in = x < g.nx && y < g.ny;
    uint32_t cmax = 0, cmin = 0, cdir = 0, bad = 0;
    uint32_t tm = 0;
    if (in) {
        const size_t i = flat(g, x, y, z);
        const uint32_t valid = valid_mask(x, y, z, g.nx, g.ny, g.nz);
        int oasc, odesc;
        K k[15];
        if (FIRST) {
            load_keys(f, i, g, valid, k);
            arg_ext(k, valid, oasc, odesc);
            codes[i] = static_cast<uint8_t>(oasc | (odesc << 4));
            bad = bad_value(f[i]) || bad_value(fh[i]);
        } else {
            const uint8_t c = codes[i];
            oasc = c & 15;
            odesc = c >> 4;
        }
        int asc, desc;
        load_keys(fh, i, g, valid, k);
        arg_ext(k, valid, asc, desc);
        tm = detect_rules(asc, desc, oasc, odesc, cmax, cmin, cdir);
        if (tm) request_targets(req, g, x, y, z, tm);
    }
    const uint32_t mism = __ballot_sync(0xFFFFFFFFu, tm != 0);
    if (threadIdx.x == 0 && y < g.ny && mism) act_next[word_of(g, blockIdx.x * 32, y, z)] = mism;
    flush_counts(slot, cmax, cmin, cdir, in ? 1u : 0u, bad);
}

// ---------------------------------------------------------------------------
// Sparse detection over the active bitmap (grid-stride over words).  The
// word's bits are consumed and cleared; mismatching voxels go to act_next
// (only this thread touches that word of act_next in this kernel).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) k_detect_sparse(const T *__restrict__ fh, const uint8_t *__restrict__ codes,
                                                       uint32_t *__restrict__ act_cur, uint32_t *__restrict__ act_next,
                                                       uint32_t *__restrict__ req, SweepSlot *slot, Geom g) {
    using K = typename KeyOf<T>::type;
    uint32_t cmax = 0, cmin = 0, cdir = 0, active = 0;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t w = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < g.nwords; w += stride) {
        uint32_t bits = act_cur[w];
        if (!bits) continue;
        act_cur[w] = 0;
        const size_t row = w / g.wpr;
        const int wx = static_cast<int>(w - row * g.wpr);
        const int y = static_cast<int>(row % g.ny);
        const int z = static_cast<int>(row / g.ny);
        uint32_t mism = 0;
        active += __popc(bits);
        while (bits) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1;
            const int x = wx * 32 + b;
            const size_t i = flat(g, x, y, z);
            const uint32_t valid = valid_mask(x, y, z, g.nx, g.ny, g.nz);
            K k[15];
            load_keys(fh, i, g, valid, k);
            int asc, desc;
            arg_ext(k, valid, asc, desc);
            const uint8_t c = codes[i];
            const uint32_t tm = detect_rules(asc, desc, c & 15, c >> 4, cmax, cmin, cdir);
            if (tm) {
                request_targets(req, g, x, y, z, tm);
                mism |= 1u << b;
            }
        }
        if (mism) act_next[w] = mism;
    }
    flush_counts(slot, cmax, cmin, cdir, active, 0);
}

// ---------------------------------------------------------------------------
// Apply: applyDeltaBuffer_local (pMSz.cu:623-645) on every requested vertex,
// in T:  if |f - (fhat - delta)| <= eps && cnt < q-1 { fhat -= delta; cnt++ }
//        else { cnt = q; fhat = f - eps }
// then mark the closed stencil of every vertex whose value changed.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) k_apply(const T *__restrict__ f, T *__restrict__ fh, uint8_t *__restrict__ cnt,
                                               uint32_t *__restrict__ req, uint32_t *__restrict__ act_next,
                                               SweepSlot *slot, Geom g, T eps, T delta, int q) {
    uint32_t nreq = 0, nchg = 0, nprog = 0;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t w = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < g.nwords; w += stride) {
        uint32_t bits = req[w];
        if (!bits) continue;
        req[w] = 0;
        const size_t row = w / g.wpr;
        const int wx = static_cast<int>(w - row * g.wpr);
        const int y = static_cast<int>(row % g.ny);
        const int z = static_cast<int>(row / g.ny);
        nreq += __popc(bits);
        uint32_t changed = 0;
        while (bits) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1;
            bool prog;
            const uint32_t c = apply_one(f, fh, cnt, flat(g, wx * 32 + b, y, z), eps, delta, q, prog);
            changed |= c << b;
            nprog += prog ? 1u : 0u;
        }
        nchg += __popc(changed);
        if (changed) mark_stencil(act_next, g, wx, y, z, changed);
    }
    nreq = warp_sum_u32(nreq);
    nchg = warp_sum_u32(nchg);
    nprog = warp_sum_u32(nprog);
    if ((threadIdx.x & 31) == 0) {
        if (nreq) atomicAdd(&slot->requested, (unsigned long long)nreq);
        if (nchg) atomicAdd(&slot->changed, (unsigned long long)nchg);
        if (nprog) atomicAdd(&slot->progressed, (unsigned long long)nprog);
    }
}

}  // namespace pmsz

#include "sweep.cuh"

namespace pmsz {

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
static inline dim3 grid3(const Geom &g) {
    return dim3(static_cast<unsigned>(g.wpr), static_cast<unsigned>((g.ny + 7) / 8), static_cast<unsigned>(g.nz));
}

static inline unsigned stride_grid(size_t items) {
    const size_t want = (items + 255) / 256;
    return static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>(want, 152 * 16)));
}

// Tensor maps of f and fhat for the TMA-fed first pass (k_pair_tma): 3-D
// (nx, ny, nz) maps with a box of one tile plane.  The encoder is the driver's
// cuTensorMapEncodeTiled, reached through the runtime (the library does not
// link libcuda).  Not available (ok = false: the first pass loads its tiles
// itself) when the encoder is missing, the fields are not 16-byte aligned or
// a row is not a multiple of 16 bytes.
struct FirstMaps {
    CUtensorMap f, fh;
    bool ok = false;
};

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

template <typename T>
static FirstMaps first_maps(const T *f, const T *fh, const Geom &g) {
    FirstMaps m;
    const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc || (static_cast<size_t>(g.nx) * sizeof(T)) % 16 || reinterpret_cast<uintptr_t>(f) % 16 ||
        reinterpret_cast<uintptr_t>(fh) % 16)
        return m;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(g.nx), static_cast<cuuint64_t>(g.ny),
                                static_cast<cuuint64_t>(g.nz)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(g.nx) * sizeof(T),
                                   static_cast<cuuint64_t>(g.nx) * g.ny * sizeof(T)};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(RawBox<T>::kX), static_cast<cuuint32_t>(kMHY), 1u};
    const cuuint32_t es[3] = {1u, 1u, 1u};
    const CUtensorMapDataType dt = sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    for (int k = 0; k < 2; ++k)
        if (enc(k ? &m.fh : &m.f, dt, 3, const_cast<T *>(k ? fh : f), dims, strides, box, es,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return m;
    m.ok = true;
    return m;
}

constexpr char kCopyMissing[] = "first pass: a tile plane's tensor copy did not arrive within the bounded wait";

// The fused first pass over the z-chunks bz0 .. bz0+grid.z-1: TMA-fed when the
// maps exist; *err is set if a plane's copy did not arrive within the bounded
// wait.
template <typename T>
static int launch_first_pass(const FirstMaps &m, dim3 grid, cudaStream_t s, const T *f, T *fh, uint8_t *codes,
                             uint32_t *hp, uint32_t *req, uint32_t *act, SweepSlot *slot, const Geom &g, int bz0,
                             uint32_t *err, uint8_t *freq = nullptr, uint8_t *fact = nullptr) {
    const MarchArgs<T> a{f, fh, codes, hp, req, act, slot, freq, fact};
    if (m.ok) {
        PMSZ_CUDA(allow_smem(k_pair_tma<T, kFirst>, sizeof(TmaMarch<T>)));
        k_pair_tma<T, kFirst><<<grid, dim3(kTX, kThreads / kTX, 1), sizeof(TmaMarch<T>), s>>>(m.f, m.fh, a, g, bz0, err);
        PMSZ_CUDA(cudaGetLastError());
    } else {
        PMSZ_CUDA((launch_march<T, kFirst>(grid, s, a, g, bz0)));
    }
    return PMSZ_OK;
}

// A sweep kernel over all resident blocks of the current device (queried once
// per device, since the queries cost more than a small field's sweep), or as
// many as `words` bitmap words keep busy.
template <typename T, class Kernel, class... Args>
static int launch_cooperative(Kernel kernel, size_t words, cudaStream_t s, const Args &...args) {
    static std::mutex mu;
    static std::vector<std::pair<unsigned, unsigned>> known;  // resident blocks; three per SM
    unsigned blocks = 0, three = 0;
    {
        int dev = 0;
        PMSZ_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        if (static_cast<size_t>(dev) >= known.size()) known.resize(static_cast<size_t>(dev) + 1, {0u, 0u});
        if (!known[static_cast<size_t>(dev)].first) {
            int sms = 0, per_sm = 0, coop = 0;
            PMSZ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            PMSZ_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
            if (!coop) return set_error(PMSZ_ERR_CUDA, "device does not support cooperative launches");
            PMSZ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSweepBlock, 0));
            if (per_sm < 1) return set_error(PMSZ_ERR_CUDA, "sweep kernel does not fit on an SM");
            known[static_cast<size_t>(dev)] = {static_cast<unsigned>(per_sm * sms), static_cast<unsigned>(3 * sms)};
        }
        std::tie(blocks, three) = known[static_cast<size_t>(dev)];
    }
    const size_t groups = (words + kGroupWords - 1) / kGroupWords, want = (groups + kSweepWarps - 1) / kSweepWarps;
    // fp32 fits four blocks per SM: they pay where every warp has eight groups
    // (512^3 1966 us with three, 1871 with four; 256^3 2844 and 2662), fields
    // below wait for their gathers less than for the larger barrier (128^3 383
    // and 400, 120x130x128 931 and 990)
    const unsigned most = groups >= 8u * kSweepWarps * static_cast<size_t>(blocks) ? blocks : std::min(blocks, three);
    const unsigned grid = static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>(want, most)));
    void *ptr[] = {const_cast<void *>(static_cast<const void *>(&args))...};
    PMSZ_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel), dim3(grid), dim3(kSweepBlock), ptr, 0, s));
    return PMSZ_OK;
}

// Grid of the list-compaction kernels: one block per 2048-word round, at most
// 16 blocks per SM (grid-stride beyond).
static inline unsigned list_grid(const Geom &g) {
    const size_t want = (g.nwords + kRoundWords - 1) / kRoundWords;
    return static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>(want, 152 * 16)));
}

int check_geom(size_t nx, size_t ny, size_t nz) {
    if (nx == 0 || ny == 0 || nz == 0) return set_error(PMSZ_ERR_ARG, "field dimensions must be positive");
    if (nx > (1u << 30) || ny > 65535 * 8 || nz > 65535)
        return set_error(PMSZ_ERR_ARG, "field dimensions exceed the supported range (nz <= 65535)");
    if (((nx + 31) / 32) * ny * nz >= (static_cast<size_t>(1) << 32))
        return set_error(PMSZ_ERR_ARG, "field too large: ceil(nx/32)*ny*nz must stay below 2^32");
    return PMSZ_OK;
}

// Slabs of the host-buffer copy: whole z-chunks, about 64 MiB of f + fhat.
// The copy of slab j ends one plane past its chunks (planes b_j .. b_{j+1} - 1
// with b_j = j * cps * zc + 1, b_0 = 0, the last ending at nz), so the first
// pass of slab j's chunks, whose tiles read one plane beyond them, waits for
// the copy of slab j only: once the host link delivers the last slab, one
// slab's first pass is left, not two.
struct IngestSlabs {
    int cps, nchunks, nslabs;
};
static IngestSlabs ingest_slabs(const Geom &g, size_t elem) {
    const size_t plane = static_cast<size_t>(g.nx) * g.ny;
    const size_t chunk_bytes = 2 * plane * static_cast<size_t>(g.zc) * elem;
    IngestSlabs r;
    r.nchunks = (g.nz + g.zc - 1) / g.zc;
    r.cps = static_cast<int>(std::max<size_t>(1, (static_cast<size_t>(64) << 20) / chunk_bytes));
    r.nslabs = (r.nchunks + r.cps - 1) / r.cps;
    return r;
}
static size_t slab_begin(int j, int cps, int nslabs, int zc, size_t nz) {
    if (j <= 0) return 0;
    if (j >= nslabs) return nz;
    return std::min(nz, static_cast<size_t>(j) * cps * zc + 1);  // j * cps * zc < nz for j < nslabs
}

template <typename T>
int enqueue_ingest(const T *hf, const T *hfh, T *df, T *dfh, T *dprev, size_t nx, size_t ny, size_t nz,
                   cudaStream_t s, IngestCopies &c) {
    int rc = check_geom(nx, ny, nz);
    if (rc) return rc;
    Geom g = make_geom(nx, ny, nz);
    // the tile depth correct_impl will use; slabs are whole columns, and the last
    // one is what is left when the copy ends, so at most 32 planes
    g.zc = std::min(first_depth(nx, ny, nz, sizeof(T)), 32);
    const IngestSlabs sl = ingest_slabs(g, sizeof(T));
    c.cps = sl.cps;
    c.nchunks = sl.nchunks;
    c.nslabs = sl.nslabs;
    c.zc = g.zc;
    const size_t plane = static_cast<size_t>(g.nx) * g.ny;
    // cs: host copies; ds: device copies of fhat into dprev (kept off cs so
    // the host link never idles behind them)
    PMSZ_CUDA(cudaStreamCreateWithFlags(&c.cs, cudaStreamNonBlocking));
    PMSZ_CUDA(cudaStreamCreateWithFlags(&c.ds, cudaStreamNonBlocking));
    c.ev.assign(static_cast<size_t>(c.nslabs) + 1, nullptr);
    c.evp.assign(static_cast<size_t>(c.nslabs), nullptr);
    for (cudaEvent_t &e : c.ev) PMSZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (cudaEvent_t &e : c.evp) PMSZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    PMSZ_CUDA(cudaEventRecord(c.ev[c.nslabs], s));  // the destinations are allocated
    PMSZ_CUDA(cudaStreamWaitEvent(c.cs, c.ev[c.nslabs], 0));
    for (int j = 0; j < c.nslabs; ++j) {
        const size_t z0 = slab_begin(j, c.cps, c.nslabs, g.zc, g.nz);
        const size_t z1 = slab_begin(j + 1, c.cps, c.nslabs, g.zc, g.nz);
        const size_t off = z0 * plane, bytes = (z1 - z0) * plane * sizeof(T);
        if (bytes) {
            PMSZ_CUDA(cudaMemcpyAsync(df + off, hf + off, bytes, cudaMemcpyHostToDevice, c.cs));
            PMSZ_CUDA(cudaMemcpyAsync(dfh + off, hfh + off, bytes, cudaMemcpyHostToDevice, c.cs));
        }
        PMSZ_CUDA(cudaEventRecord(c.ev[j], c.cs));
        if (dprev) {  // the pre-correction copy of fhat, before any edit of the slab
            PMSZ_CUDA(cudaStreamWaitEvent(c.ds, c.ev[j], 0));
            if (bytes)
                PMSZ_CUDA(cudaMemcpyAsync(dprev + off, dfh + off, bytes, cudaMemcpyDeviceToDevice, c.ds));
            PMSZ_CUDA(cudaEventRecord(c.evp[j], c.ds));
        } else {
            PMSZ_CUDA(cudaEventRecord(c.evp[j], c.cs));
        }
    }
    return PMSZ_OK;
}

// The fused first pass over a field that is still being copied in from the
// host (the copies of enqueue_ingest): the first pass of a slab's chunks waits
// for that slab's event (its copy includes the plane beyond the chunks).
template <typename T>
int first_pass_ingest(const HostIngest<T> &in, const T *f, T *fh, uint8_t *codes, uint32_t *hp, uint32_t *req,
                      uint32_t *a_next, SweepSlot *slot, const Geom &g, cudaStream_t s, int64_t *launches,
                      const FirstMaps &maps, uint32_t *err, uint8_t *freq, uint8_t *fact) {
    if (in.df != f || !in.copies || in.copies->zc != g.zc)
        return set_error(PMSZ_ERR_ARG, "ingest copies do not match the field");
    const IngestCopies &r = *in.copies;
    const int cps = r.cps, nchunks = r.nchunks, nslabs = r.nslabs;
    int rc;
    for (int j = 0; j < nslabs; ++j) {
        PMSZ_CUDA(cudaStreamWaitEvent(s, r.ev[j], 0));
        dim3 grid = tiled_grid(g);
        grid.z = static_cast<unsigned>(std::min(cps, nchunks - j * cps));
        if ((rc = launch_first_pass<T>(maps, grid, s, f, fh, codes, hp, req, a_next, slot, g, j * cps, err, freq, fact))) return rc;
        PMSZ_CUDA(cudaGetLastError());
        ++*launches;
    }
    PMSZ_CUDA(cudaStreamWaitEvent(s, r.evp[nslabs - 1], 0));  // dprev complete before the first edit
    return PMSZ_OK;
}

// The fractions of the slabs after which the sweeps behind the host copy
// (kWaveSweeps of them) advance, in sixteenths.  A wave costs its launch and two
// barriers a sweep whatever its size, and dense sweeps are less efficient in
// pieces, so the first ones are large; the last ones, all that is left once the
// copy ends, are small.  256x320x288 and 512^3 fp64: 2521 us and 11.46 ms; at
// 4, 8, 12, 14, 16: 2538 and 11.64; at 12, 15, 16: 2626 and 11.51; without waves
// 2718 and 13.02.  (As voxel lists, seven launches a piece: 3347 us and 11.80.)
// With what the sweeps have gained since, 2410 us (up to 2680 from run to run) and
// 11.35 ms.
constexpr int kWaveAt[] = {8, 12, 14, 15, 16};
static_assert(std::size(kWaveAt) < std::size(LoopState{}.bar), "a barrier counter for each");

// The host-buffer wavefront.  The copy of slab j releases the first pass
// of slab j (sweep 0's detection, complete below plane Z = (j + 1) * slab
// depth, or nz after the last slab); after the slabs of kWaveAt
// follows a wave: on the planes already final, the pieces of sweeps 0 .. K that those
// planes allow:
//   sweep k's detection covers planes below D_k, its edits planes below A_k,
//   with D_0 = Z, A_k = D_k - 1 and D_k = A_{k-1} - 1 (k >= 1),
// every front reaching nz after the last slab.  Sweep k's detection reads
// planes up to D_k = A_{k-1} - 1, all edited by sweep k - 1 already; its
// edits stop one plane below D_k, so no later detection of sweep k reads an
// edited plane or requests an edit below A_k; the active set of sweep k + 1
// below D_{k+1} is final once sweep k has edited planes up to D_{k+1} + 1.
// Each sweep thus sees exactly the field, codes and active set of the
// snapshot schedule, and sweeps that run while the rest of the field is still
// crossing the host link leave little to do after it.  Counters go straight
// to slots[k]; k_wave_gate then sets the loop state as after sweep K.
template <typename T>
static int first_pass_waves(const HostIngest<T> &in, const SweepArgs<T> &a, const FirstMaps &maps, int K, cudaStream_t s,
                            int64_t *launches) {
    const Geom &g = a.g;
    if (in.df != a.f || !in.copies || in.copies->zc != g.zc)
        return set_error(PMSZ_ERR_ARG, "ingest copies do not match the field");
    const IngestCopies &r = *in.copies;
    const int cps = r.cps, nchunks = r.nchunks, nslabs = r.nslabs;
    const uint32_t plane_words = static_cast<uint32_t>(static_cast<size_t>(g.wpr) * g.ny);  // (nwords < 2^32)
    int rc;
    WaveFronts f{};
    f.sweeps = K;
    std::vector<int> Dp(static_cast<size_t>(K) + 1, 0), Ap(static_cast<size_t>(K) + 1, 0);  // fronts so far, in planes
    std::vector<char> wave_after(static_cast<size_t>(nslabs), 0);
    for (int e : kWaveAt) wave_after[static_cast<size_t>(std::max(1, (nslabs * e + 15) / 16) - 1)] = 1;
    for (int j = 0; j < nslabs; ++j) {
        const bool last = j == nslabs - 1;
        PMSZ_CUDA(cudaStreamWaitEvent(s, r.ev[j], 0));
        dim3 grid = tiled_grid(g);
        grid.z = static_cast<unsigned>(std::min(cps, nchunks - j * cps));
        if ((rc = launch_first_pass<T>(maps, grid, s, a.f, a.fh, const_cast<uint8_t *>(a.codes), a.hp, a.req, a.act1,
                                       &a.slots[0], g, j * cps, &a.ls->err, a.freq, a.f1)))
            return rc;
        ++*launches;
        if (!wave_after[static_cast<size_t>(j)]) continue;
        PMSZ_CUDA(cudaStreamWaitEvent(s, r.evp[j], 0));  // fhat's pre-correction copy of slabs 0 .. j
        const int Z = last ? g.nz : std::min(g.nz, (j + 1) * cps * g.zc);
        size_t widest = 0;
        for (int k = 0; k <= K; ++k) {
            const int D = last ? g.nz : std::max(Dp[k], k == 0 ? Z : Ap[k - 1] - 1);
            f.det0[k] = plane_words * static_cast<uint32_t>(Dp[k]);
            f.det1[k] = plane_words * static_cast<uint32_t>(D);
            Dp[k] = D;
            const int A = last ? g.nz : std::max(Ap[k], D - 1);
            f.edit0[k] = plane_words * static_cast<uint32_t>(Ap[k]);
            f.edit1[k] = plane_words * static_cast<uint32_t>(A);
            Ap[k] = A;
            widest = std::max<size_t>(widest, std::max(f.det1[k] - f.det0[k], f.edit1[k] - f.edit0[k]));
        }
        ++f.launch;
        if ((rc = launch_cooperative<T>(k_sweep_wave<T>, widest, s, a, f))) return rc;
        ++*launches;
    }
    return PMSZ_OK;
}

template int enqueue_ingest<float>(const float *, const float *, float *, float *, float *, size_t, size_t, size_t,
                                   cudaStream_t, IngestCopies &);
template int enqueue_ingest<double>(const double *, const double *, double *, double *, double *, size_t, size_t,
                                    size_t, cudaStream_t, IngestCopies &);

template <typename T>
int correct_impl(const T *f, T *fh, size_t nx, size_t ny, size_t nz, double eb, const pmsz_opts *opts,
                 pmsz_result *res, cudaStream_t s, const HostIngest<T> *ingest) {
    if (!f || !fh) return set_error(PMSZ_ERR_ARG, "null field pointer");
    int rc = check_geom(nx, ny, nz);
    if (rc) return rc;
    const int q = opts ? opts->q : 5;
    const uint32_t flags = opts ? opts->flags : 0u;
    const int64_t max_sweeps = opts && opts->max_sweeps > 0 ? opts->max_sweeps : 10000;
    if (!(eb > 0.0) || !(eb < 1e300)) return set_error(PMSZ_ERR_ARG, "error bound must be positive and finite");
    if (q < 1 || q > 255) return set_error(PMSZ_ERR_ARG, "q must be in 1..255");
    if ((flags & PMSZ_FLAG_AUTOTUNE) && !ingest && !tune_known(nx, ny, nz, sizeof(T)) &&
        (rc = autotune_impl<T>(f, fh, nx, ny, nz, nullptr, s)))
        return rc;
    Geom g = make_geom(nx, ny, nz);
    g.zc = ingest && ingest->copies ? ingest->copies->zc : first_depth(nx, ny, nz, sizeof(T));
    const T eps = static_cast<T>(eb);
    const T delta = static_cast<T>(eb / static_cast<double>(q));  // pMSz.cu:2814

    // Scratch: what starts at zero first, in one piece (loop state and sweep
    // slots, counters, request + two active bitmaps with their group flags),
    // then codes and proxies.
    const bool full = (flags & PMSZ_FLAG_FULL_SWEEPS) != 0;
    const size_t groups = group_count(g);
    Workspace ws(s);
    const size_t o_ls = ws.reserve<LoopState>(1);
    const size_t o_slots = ws.reserve<SweepSlot>(static_cast<size_t>(max_sweeps));
    const bool own_cnt = !(ingest && ingest->cnt);
    const size_t o_cnt = ws.reserve<uint8_t>(own_cnt ? g.n : 0);
    const size_t o_req = ws.reserve<uint32_t>(g.nwords);
    const size_t o_a0 = ws.reserve<uint32_t>(g.nwords);
    const size_t o_a1 = ws.reserve<uint32_t>(g.nwords);
    const size_t o_fr = ws.reserve<uint8_t>(groups), o_f0 = ws.reserve<uint8_t>(groups), o_f1 = ws.reserve<uint8_t>(groups);
    const size_t zero_bytes = ws.reserve<uint8_t>(0);
    const size_t o_codes = ws.reserve<uint8_t>(g.n);
    constexpr bool proxies = sizeof(T) == 8;  // (fp32 sweeps compare the values themselves)
    const size_t o_hp = ws.reserve<uint32_t>(proxies ? g.n : 0);
    // host-buffer calls of several slabs run sweeps 1 .. K behind the copy
    // (first_pass_waves; K below max_sweeps)
    const int wave_k = static_cast<int>(std::min<int64_t>(kWaveSweeps, max_sweeps - 1));
    const bool waves = ingest && !full && wave_k >= 1 && ingest->copies &&
                       ingest->copies->nslabs >= 2;
    if ((rc = ws.commit())) return rc;
    LoopState *ls = ws.at<LoopState>(o_ls);
    SweepSlot *slots = ws.at<SweepSlot>(o_slots);
    uint8_t *cnt = own_cnt ? ws.at<uint8_t>(o_cnt) : ingest->cnt;
    uint32_t *req = ws.at<uint32_t>(o_req);
    uint32_t *act[2] = {ws.at<uint32_t>(o_a0), ws.at<uint32_t>(o_a1)};
    uint8_t *freq = ws.at<uint8_t>(o_fr), *fact[2] = {ws.at<uint8_t>(o_f0), ws.at<uint8_t>(o_f1)};
    uint8_t *codes = ws.at<uint8_t>(o_codes);
    uint32_t *hp = proxies ? ws.at<uint32_t>(o_hp) : nullptr;
    const FirstMaps maps = first_maps<T>(f, fh, g);
    EventTimer et;
    if ((rc = et.init())) return rc;
    PMSZ_CUDA(cudaEventRecord(et.ev[3], s));  // start of the loop's device window

    PMSZ_CUDA(cudaMemsetAsync(ls, 0, zero_bytes, s));  // init_counter among them, pMSz.cu:1745-1749
    if (!own_cnt) PMSZ_CUDA(cudaMemsetAsync(cnt, 0, g.n, s));

    const bool timing = (flags & PMSZ_FLAG_TIMING) != 0;
    double ms_first = 0, ms_detect = 0, ms_apply = 0;
    int64_t launches = 0;
    int64_t sweeps = 0;
    uint64_t edits = 0;
    int status = PMSZ_ERR_NOT_CONVERGED;
    bool end_recorded = false;  // et.ev[0] marks the end of the correction's device window
    std::vector<SweepSlot> log;
    // The state and the first slots of the sweep log, in one read-back.
    constexpr int64_t kLogAhead = 64;
    static_assert(sizeof(LoopState) <= 256, "the slots follow the loop state at its 256-byte slot");
    const int64_t pre = std::min<int64_t>(max_sweeps, kLogAhead);
    const size_t head = 256 + static_cast<size_t>(pre) * sizeof(SweepSlot);
    unsigned char *hb = static_cast<unsigned char *>(host_pinned(head));
    if (!hb) return set_error(PMSZ_ERR_OOM, "pinned host allocation failed");
    const LoopState *hls = reinterpret_cast<const LoopState *>(hb);
    const SweepSlot *hlog = reinterpret_cast<const SweepSlot *>(hb + 256);
    if (!full) {
        // The fused first pass, then every sweep in one cooperative launch
        // (k_sweeps), which starts with the edits of sweep 0 -- or, behind the
        // host copy, where the wavefront left off.  One read-back at the end.
        EventTimer lt;  // start, first pass done, sweeps done
        if (timing) {
            if ((rc = lt.init())) return rc;
            PMSZ_CUDA(cudaEventRecord(lt.ev[0], s));
        }
        SweepArgs<T> a{f,  fh,         codes, cnt, hp,  req,   act[0], act[1], freq, fact[0], fact[1], slots,
                       ls, max_sweeps, 1,     g,   eps, delta, q};
        if (waves) {
            if ((rc = first_pass_waves<T>(*ingest, a, maps, wave_k, s, &launches))) return rc;
            k_wave_gate<<<1, 32, 0, s>>>(ls, slots, wave_k, max_sweeps);
            PMSZ_CUDA(cudaGetLastError());
            ++launches;
            a.from_edits = 0;
        } else if (ingest) {
            if ((rc = first_pass_ingest<T>(*ingest, f, fh, codes, hp, req, act[1], &slots[0], g, s, &launches,
                                           maps, &ls->err, freq, fact[1])))
                return rc;
        } else {
            if ((rc = launch_first_pass<T>(maps, tiled_grid(g), s, f, fh, codes, hp, req, act[1], &slots[0], g, 0,
                                           &ls->err, freq, fact[1])))
                return rc;
            ++launches;
        }
        if (timing) PMSZ_CUDA(cudaEventRecord(lt.ev[1], s));
        if ((rc = launch_cooperative<T>(k_sweeps<T>, g.nwords, s, a))) return rc;
        ++launches;
        if (timing) PMSZ_CUDA(cudaEventRecord(lt.ev[2], s));
        PMSZ_CUDA(cudaEventRecord(et.ev[0], s));  // end of the correction's device window
        end_recorded = true;
        PMSZ_CUDA(cudaMemcpyAsync(hb, ls, head, cudaMemcpyDeviceToHost, s));
        if (ingest && ingest->after && ingest->after->fn) {
            ingest->after->done = true;
            if ((rc = ingest->after->fn(s))) return rc;
        }
        PMSZ_CUDA(cudaStreamSynchronize(s));
        if (hls->err) return set_error(PMSZ_ERR_CUDA, hls->err & kErrCopy ? kCopyMissing : kBarrierMissing);
        const int64_t done = hls->done;  // sweeps 0 .. done-1
        if (timing) {  // sweep 0's edits run inside the launch and count as detection time
            float x = 0, y = 0;
            PMSZ_CUDA(cudaEventElapsedTime(&x, lt.ev[0], lt.ev[1]));
            PMSZ_CUDA(cudaEventElapsedTime(&y, lt.ev[1], lt.ev[2]));
            ms_first += x;
            ms_detect += y;
        }
        log.assign(hlog, hlog + std::min(done, pre));
        if (done > pre) {
            log.resize(static_cast<size_t>(done));
            PMSZ_CUDA(cudaMemcpyAsync(log.data() + pre, slots + pre, static_cast<size_t>(done - pre) * sizeof(SweepSlot),
                                      cudaMemcpyDeviceToHost, s));
            PMSZ_CUDA(cudaStreamSynchronize(s));
        }
        for (const SweepSlot &t : log) edits += t.requested;
        sweeps = done;
        const SweepSlot &last = log.back();
        if (done == 1 && last.bad) {
            status = set_error(PMSZ_ERR_ARG, "input contains NaN or the value 1e30 (the reference's halo sentinel)");
        } else if (last.fmax == 0 && last.fmin == 0 && last.fdir == 0) {
            status = PMSZ_OK;
        } else if (last.progressed == 0) {
            set_error(PMSZ_ERR_NOT_CONVERGED, "a sweep requested edits that changed nothing (all requested vertices clamped)");
        }
    }
    // The reference's schedule: every sweep over the whole field, host-driven.
    while (full && sweeps < max_sweeps) {
        SweepSlot *slot = slots + sweeps;
        if (timing) PMSZ_CUDA(cudaEventRecord(et.ev[0], s));
        if (sweeps == 0 && ingest) {
            if ((rc = first_pass_ingest<T>(*ingest, f, fh, codes, hp, req, act[1], slot, g, s, &launches, maps,
                                           &ls->err, nullptr, nullptr)))
                return rc;
        } else if (sweeps == 0) {
            if ((rc = launch_first_pass<T>(maps, tiled_grid(g), s, f, fh, codes, hp, req, act[1], slot, g, 0,
                                           &ls->err)))
                return rc;
            ++launches;
        } else {
            PMSZ_CUDA((launch_field<T, kDetect>(s, MarchArgs<T>{nullptr, fh, codes, nullptr, req, nullptr, slot}, g)));
            ++launches;
        }
        if (timing) PMSZ_CUDA(cudaEventRecord(et.ev[1], s));
        k_apply_full<T><<<list_grid(g), kListBlock, 0, s>>>(f, fh, cnt, req, slot, g, eps, delta, q);
        ++launches;
        if (timing) PMSZ_CUDA(cudaEventRecord(et.ev[2], s));
        PMSZ_CUDA(cudaGetLastError());
        SweepSlot *hslot = reinterpret_cast<SweepSlot *>(hb + 256);
        PMSZ_CUDA(cudaMemcpyAsync(hslot, slot, sizeof(SweepSlot), cudaMemcpyDeviceToHost, s));
        if (sweeps == 0) PMSZ_CUDA(cudaMemcpyAsync(hb, ls, sizeof(LoopState), cudaMemcpyDeviceToHost, s));
        PMSZ_CUDA(cudaStreamSynchronize(s));
        if (sweeps == 0 && hls->err) return set_error(PMSZ_ERR_CUDA, kCopyMissing);
        if (timing) {
            float x = 0, y = 0;
            PMSZ_CUDA(cudaEventElapsedTime(&x, et.ev[0], et.ev[1]));
            PMSZ_CUDA(cudaEventElapsedTime(&y, et.ev[1], et.ev[2]));
            (sweeps == 0 ? ms_first : ms_detect) += x;
            ms_apply += y;
        }
        ++sweeps;
        const SweepSlot h = *hslot;
        log.push_back(h);
        edits += h.requested;
        if (sweeps == 1 && h.bad) {
            status = set_error(PMSZ_ERR_ARG, "input contains NaN or the value 1e30 (the reference's halo sentinel)");
            break;
        }
        if (h.fmax == 0 && h.fmin == 0 && h.fdir == 0) { status = PMSZ_OK; break; }
        if (h.progressed == 0) {
            set_error(PMSZ_ERR_NOT_CONVERGED, "a sweep requested edits that changed nothing (all requested vertices clamped)");
            break;
        }
    }
    float ms_total = 0;
    if (!end_recorded) PMSZ_CUDA(cudaEventRecord(et.ev[0], s));
    PMSZ_CUDA(cudaEventSynchronize(et.ev[0]));
    PMSZ_CUDA(cudaEventElapsedTime(&ms_total, et.ev[3], et.ev[0]));
    if (status == PMSZ_ERR_NOT_CONVERGED && sweeps >= max_sweeps)
        set_error(PMSZ_ERR_NOT_CONVERGED, "max_sweeps reached before convergence");
    if (res) {
        res->sweeps = sweeps;
        res->iteration = sweeps + 1;
        res->edits = edits;
        res->ms_first_pass = ms_first;
        res->ms_detect = ms_detect;
        res->ms_apply = ms_apply;
        res->launches = launches;
        res->ms_total = ms_total;
        if (res->sweep_log && res->sweep_log_cap > 0) {
            const size_t m = std::min<size_t>(log.size(), static_cast<size_t>(res->sweep_log_cap));
            static_assert(sizeof(SweepSlot) == sizeof(pmsz_sweep_record), "record layout");
            std::memcpy(res->sweep_log, log.data(), m * sizeof(SweepSlot));
        }
    }
    rc = ws.release();
    return status != PMSZ_OK ? status : rc;
}

template <typename T>
int codes_impl(const T *v, size_t nx, size_t ny, size_t nz, uint8_t *codes, cudaStream_t s) {
    if (!v || !codes) return set_error(PMSZ_ERR_ARG, "null pointer");
    int rc = check_geom(nx, ny, nz);
    if (rc) return rc;
    Geom g = make_geom(nx, ny, nz);
    g.zc = first_depth(nx, ny, nz, sizeof(T));
    PMSZ_CUDA((launch_field<T, kCodes>(s, MarchArgs<T>{v, nullptr, codes, nullptr, nullptr, nullptr, nullptr}, g)));
    PMSZ_CUDA(cudaGetLastError());
    return PMSZ_OK;
}

// Both fields' codes in one pass, their differences and the values' distances
// counted (MarchArgs::pair); *err as in the first pass.
template <typename T>
int pair_impl(const T *f, const T *fp, size_t nx, size_t ny, size_t nz, T eps, uint64_t sure, uint8_t *c0, uint8_t *c1,
              unsigned long long *counts, uint32_t *err, cudaStream_t s) {
    Geom g = make_geom(nx, ny, nz);
    g.zc = first_depth(nx, ny, nz, sizeof(T));
    MarchArgs<T> a{f, fp, c0, nullptr, nullptr, nullptr, nullptr};
    a.codes_h = c1;
    a.eps = eps;
    a.sure = sure;
    a.pair = counts;
    const FirstMaps m = first_maps<T>(f, fp, g);
    if (m.ok) {
        PMSZ_CUDA(allow_smem(k_pair_tma<T, kPair>, sizeof(TmaMarch<T>)));
        k_pair_tma<T, kPair><<<tiled_grid(g), dim3(kTX, kThreads / kTX, 1), sizeof(TmaMarch<T>), s>>>(m.f, m.fh, a, g, 0, err);
        PMSZ_CUDA(cudaGetLastError());
    } else {
        PMSZ_CUDA((launch_march<T, kPair>(tiled_grid(g), s, a, g, 0)));
    }
    return PMSZ_OK;
}
template int pair_impl<float>(const float *, const float *, size_t, size_t, size_t, float, uint64_t, uint8_t *, uint8_t *,
                              unsigned long long *, uint32_t *, cudaStream_t);
template int pair_impl<double>(const double *, const double *, size_t, size_t, size_t, double, uint64_t, uint8_t *,
                               uint8_t *, unsigned long long *, uint32_t *, cudaStream_t);

// The tuner's first-pass timing: the fused first pass of f / fhat at each
// tile depth zcs[k] on scratch of its own; ms[k] is the best of two timed
// launches after a warm-up.  The code bytes (independent of the depth) go to
// the caller's buffer.
template <typename T>
int time_first_pass(const T *f, const T *fh, size_t nx, size_t ny, size_t nz, uint8_t *codes, const int *zcs, int m,
                    float *ms, cudaStream_t s) {
    Geom g = make_geom(nx, ny, nz);
    Workspace ws(s);
    const size_t o_hp = ws.reserve<uint32_t>(sizeof(T) == 8 ? g.n : 0), o_req = ws.reserve<uint32_t>(g.nwords),
                 o_act = ws.reserve<uint32_t>(g.nwords), o_slot = ws.reserve<SweepSlot>(1),
                 o_err = ws.reserve<uint32_t>(1);
    int rc = ws.commit();
    if (rc) return rc;
    const FirstMaps maps = first_maps<T>(f, fh, g);
    uint32_t *hp = sizeof(T) == 8 ? ws.at<uint32_t>(o_hp) : nullptr;  // as a correction runs it
    uint32_t *req = ws.at<uint32_t>(o_req), *act = ws.at<uint32_t>(o_act);
    uint32_t *err = ws.at<uint32_t>(o_err);
    SweepSlot *slot = ws.at<SweepSlot>(o_slot);
    PMSZ_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), s));
    EventTimer et;
    if ((rc = et.init())) return rc;
    for (int k = 0; k < m; ++k) {
        g.zc = march_depth(zcs[k]);
        float best = 0.f;
        for (int rep = 0; rep < 3; ++rep) {  // the first run of each candidate is a warm-up
            PMSZ_CUDA(cudaMemsetAsync(req, 0, g.nwords * 4, s));
            PMSZ_CUDA(cudaMemsetAsync(act, 0, g.nwords * 4, s));
            PMSZ_CUDA(cudaMemsetAsync(slot, 0, sizeof(SweepSlot), s));
            PMSZ_CUDA(cudaEventRecord(et.ev[0], s));
            if ((rc = launch_first_pass<T>(maps, tiled_grid(g), s, f, const_cast<T *>(fh), codes, hp, req, act, slot, g, 0,
                                               err)))
                return rc;
            PMSZ_CUDA(cudaGetLastError());
            PMSZ_CUDA(cudaEventRecord(et.ev[1], s));
            PMSZ_CUDA(cudaEventSynchronize(et.ev[1]));
            float t = 0.f;
            PMSZ_CUDA(cudaEventElapsedTime(&t, et.ev[0], et.ev[1]));
            if (rep > 0 && (best == 0.f || t < best)) best = t;
        }
        ms[k] = best;
    }
    uint32_t herr = 0;
    PMSZ_CUDA(cudaMemcpyAsync(&herr, err, sizeof(herr), cudaMemcpyDeviceToHost, s));
    PMSZ_CUDA(cudaStreamSynchronize(s));
    if (herr) return set_error(PMSZ_ERR_CUDA, kCopyMissing);
    return ws.release();
}

template int time_first_pass<float>(const float *, const float *, size_t, size_t, size_t, uint8_t *, const int *, int,
                                    float *, cudaStream_t);
template int time_first_pass<double>(const double *, const double *, size_t, size_t, size_t, uint8_t *, const int *,
                                     int, float *, cudaStream_t);

template int codes_impl<float>(const float *, size_t, size_t, size_t, uint8_t *, cudaStream_t);
template int codes_impl<double>(const double *, size_t, size_t, size_t, uint8_t *, cudaStream_t);

template int correct_impl<float>(const float *, float *, size_t, size_t, size_t, double, const pmsz_opts *, pmsz_result *, cudaStream_t, const HostIngest<float> *);
template int correct_impl<double>(const double *, double *, size_t, size_t, size_t, double, const pmsz_opts *, pmsz_result *, cudaStream_t, const HostIngest<double> *);

}  // namespace pmsz

using namespace pmsz;

extern "C" int pmsz_correct_f32(const float *f, float *fhat, size_t nx, size_t ny, size_t nz, double eb,
                                const pmsz_opts *opts, pmsz_result *res, void *stream) {
    return guarded([&] { return correct_impl<float>(f, fhat, nx, ny, nz, eb, opts, res, as_stream(stream)); });
}
extern "C" int pmsz_correct_f64(const double *f, double *fhat, size_t nx, size_t ny, size_t nz, double eb,
                                const pmsz_opts *opts, pmsz_result *res, void *stream) {
    return guarded([&] { return correct_impl<double>(f, fhat, nx, ny, nz, eb, opts, res, as_stream(stream)); });
}
extern "C" int pmsz_codes_f32(const float *v, size_t nx, size_t ny, size_t nz, uint8_t *codes, void *stream) {
    return guarded([&] { return codes_impl<float>(v, nx, ny, nz, codes, as_stream(stream)); });
}
extern "C" int pmsz_codes_f64(const double *v, size_t nx, size_t ny, size_t nz, uint8_t *codes, void *stream) {
    return guarded([&] { return codes_impl<double>(v, nx, ny, nz, codes, as_stream(stream)); });
}
extern "C" int pmsz_rank_offset(int r, int *dx, int *dy, int *dz) {
    if (r < 0 || r > 14 || !dx || !dy || !dz) return PMSZ_ERR_ARG;
    *dx = rank_dx(r);
    *dy = rank_dy(r);
    *dz = rank_dz(r);
    return PMSZ_OK;
}

// ---------------------------------------------------------------------------
// pmsz_correct_noalloc: the correction loop with its scratch in a fixed
// device array instead of per-call allocations, for callers that must not
// allocate device memory -- code that runs while another component owns the
// GPU's memory through its own pool or arena (a simulation that reserved HBM
// up front for in-situ compression, a serving process with a fixed budget),
// or that cannot afford an allocator call on its path.  The array below is
// part of the library image: every GPU that loads the library holds its
// PMSZ_NOALLOC_SCRATCH_BYTES until the process exits, and all calls on a
// device share it.
// ---------------------------------------------------------------------------
namespace pmsz {
namespace noalloc {

constexpr size_t kMaxVoxels = PMSZ_NOALLOC_MAX_VOXELS;
constexpr size_t kMaxWords = PMSZ_NOALLOC_MAX_WORDS;
constexpr size_t kMaxSweeps = PMSZ_NOALLOC_MAX_SWEEPS;
constexpr size_t kOffCodes = 0;
constexpr size_t kOffCnt = kOffCodes + kMaxVoxels;
constexpr size_t kOffReq = kOffCnt + kMaxVoxels;
constexpr size_t kOffAct0 = kOffReq + 4 * kMaxWords;
constexpr size_t kOffAct1 = kOffAct0 + 4 * kMaxWords;
constexpr size_t kOffSlots = kOffAct1 + 4 * kMaxWords;
constexpr size_t kBytes = kOffSlots + sizeof(SweepSlot) * kMaxSweeps;
static_assert(kBytes == PMSZ_NOALLOC_SCRATCH_BYTES, "header constant out of date");
static_assert(kOffReq % 256 == 0 && kOffSlots % 256 == 0, "sub-arrays stay 256-byte aligned");

// codes | edit counters | request bitmap | two active bitmaps | sweep slots
static __device__ __align__(256) unsigned char g_scratch[kBytes];

// Device address of g_scratch in the calling thread's current context.  The
// host-side symbol is only a stand-in for the array, so the address is looked
// up with cudaGetSymbolAddress (which allocates nothing) on every call: a
// cached address would go stale after cudaDeviceReset or in another context
// on the same device, where the library's device code is loaded again.
static int scratch_address(unsigned char **out) {
    void *p = nullptr;
    PMSZ_CUDA(cudaGetSymbolAddress(&p, g_scratch));
    *out = static_cast<unsigned char *>(p);
    return PMSZ_OK;
}

template <typename T>
int run(const T *f, T *fh, size_t nx, size_t ny, size_t nz, double eb, const pmsz_opts *opts, pmsz_result *res,
        cudaStream_t s) {
    if (!f || !fh) return set_error(PMSZ_ERR_ARG, "null field pointer");
    int rc = check_geom(nx, ny, nz);
    if (rc) return rc;
    const int q = opts ? opts->q : 5;
    const uint32_t flags = opts ? opts->flags : 0u;
    const int64_t max_sweeps = opts && opts->max_sweeps > 0 ? opts->max_sweeps : static_cast<int64_t>(kMaxSweeps);
    if (!(eb > 0.0) || !(eb < 1e300)) return set_error(PMSZ_ERR_ARG, "error bound must be positive and finite");
    if (q < 1 || q > 255) return set_error(PMSZ_ERR_ARG, "q must be in 1..255");
    const Geom g = make_geom(nx, ny, nz);
    if (g.n > kMaxVoxels)
        return set_error(PMSZ_ERR_ARG, "pmsz_correct_noalloc: field of " + std::to_string(g.n) +
                                           " voxels exceeds its fixed scratch (at most " + std::to_string(kMaxVoxels) +
                                           " voxels); use pmsz_correct_f32/f64");
    if (g.nwords > kMaxWords)
        return set_error(PMSZ_ERR_ARG, "pmsz_correct_noalloc: ceil(nx/32)*ny*nz = " + std::to_string(g.nwords) +
                                           " exceeds its fixed bitmap scratch (at most " + std::to_string(kMaxWords) + ")");
    if (max_sweeps > static_cast<int64_t>(kMaxSweeps))
        return set_error(PMSZ_ERR_ARG, "pmsz_correct_noalloc: max_sweeps above " + std::to_string(kMaxSweeps));
    unsigned char *base = nullptr;
    if ((rc = scratch_address(&base))) return rc;
    uint8_t *codes = base + kOffCodes;
    uint8_t *cnt = base + kOffCnt;
    uint32_t *req = reinterpret_cast<uint32_t *>(base + kOffReq);
    uint32_t *act[2] = {reinterpret_cast<uint32_t *>(base + kOffAct0), reinterpret_cast<uint32_t *>(base + kOffAct1)};
    SweepSlot *slots = reinterpret_cast<SweepSlot *>(base + kOffSlots);

    // The array keeps the previous call's contents: clear everything that
    // the loop expects to start at zero (codes are fully rewritten by sweep 1).
    PMSZ_CUDA(cudaMemsetAsync(cnt, 0, g.n, s));
    PMSZ_CUDA(cudaMemsetAsync(req, 0, g.nwords * 4, s));
    PMSZ_CUDA(cudaMemsetAsync(act[0], 0, g.nwords * 4, s));
    PMSZ_CUDA(cudaMemsetAsync(act[1], 0, g.nwords * 4, s));
    PMSZ_CUDA(cudaMemsetAsync(slots, 0, sizeof(SweepSlot) * static_cast<size_t>(max_sweeps), s));
    // ms_total: host clock from here to the last sweep's read-back; the loop
    // synchronises the stream after every sweep, so this is the device window
    // of the loop (timing events are not created: they are driver resources)
    PMSZ_CUDA(cudaStreamSynchronize(s));
    const auto t0 = std::chrono::steady_clock::now();

    const T eps = static_cast<T>(eb);
    const T delta = static_cast<T>(eb / static_cast<double>(q));
    const dim3 blk3(32, 8, 1);
    int cur = 0;
    int64_t sweeps = 0;
    uint64_t edits = 0;
    int status = PMSZ_ERR_NOT_CONVERGED;
    while (sweeps < max_sweeps) {
        SweepSlot *slot = slots + sweeps;
        uint32_t *a_next = act[cur ^ 1];
        if (sweeps == 0) {
            k_detect_full<T, true><<<grid3(g), blk3, 0, s>>>(f, fh, codes, req, a_next, slot, g);
        } else if (flags & PMSZ_FLAG_FULL_SWEEPS) {
            k_detect_full<T, false><<<grid3(g), blk3, 0, s>>>(nullptr, fh, codes, req, a_next, slot, g);
        } else {
            k_detect_sparse<T><<<stride_grid(g.nwords), 256, 0, s>>>(fh, codes, act[cur], a_next, req, slot, g);
        }
        k_apply<T><<<stride_grid(g.nwords), 256, 0, s>>>(f, fh, cnt, req, a_next, slot, g, eps, delta, q);
        PMSZ_CUDA(cudaGetLastError());
        SweepSlot h;  // read back into the caller's stack: no pinned buffer
        PMSZ_CUDA(cudaMemcpyAsync(&h, slot, sizeof(SweepSlot), cudaMemcpyDeviceToHost, s));
        PMSZ_CUDA(cudaStreamSynchronize(s));
        if (res && res->sweep_log && sweeps < res->sweep_log_cap)
            std::memcpy(res->sweep_log + sweeps, &h, sizeof(SweepSlot));
        ++sweeps;
        edits += h.requested;
        if (sweeps == 1 && h.bad) {
            status = set_error(PMSZ_ERR_ARG, "input contains NaN or the value 1e30 (the reference's halo sentinel)");
            break;
        }
        if (h.fmax == 0 && h.fmin == 0 && h.fdir == 0) { status = PMSZ_OK; break; }
        if (h.progressed == 0) {
            set_error(PMSZ_ERR_NOT_CONVERGED, "a sweep requested edits that changed nothing (all requested vertices clamped)");
            break;
        }
        cur ^= 1;
    }
    if (status == PMSZ_ERR_NOT_CONVERGED && sweeps >= max_sweeps)
        set_error(PMSZ_ERR_NOT_CONVERGED, "max_sweeps reached before convergence");
    if (res) {
        res->sweeps = sweeps;
        res->iteration = sweeps + 1;
        res->edits = edits;
        res->ms_first_pass = res->ms_detect = res->ms_apply = 0.0;
        res->ms_total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        res->launches = 2 * sweeps;
    }
    return status;
}

}  // namespace noalloc
}  // namespace pmsz

extern "C" int pmsz_correct_noalloc(const void *f, void *fhat, size_t elem_size, size_t nx, size_t ny, size_t nz,
                                    double eb, const pmsz_opts *opts, pmsz_result *res, void *stream) {
    return guarded([&] {
        if (elem_size == sizeof(float))
            return noalloc::run<float>(static_cast<const float *>(f), static_cast<float *>(fhat), nx, ny, nz, eb,
                                       opts, res, as_stream(stream));
        if (elem_size == sizeof(double))
            return noalloc::run<double>(static_cast<const double *>(f), static_cast<double *>(fhat), nx, ny, nz, eb,
                                        opts, res, as_stream(stream));
        return set_error(PMSZ_ERR_ARG, "elem_size must be 4 (float) or 8 (double)");
    });
}
