// batch.cu -- many independent fields corrected together.
//
// pmsz_correct_batch runs the correction of every field of a batch with one
// set of launches: the fused labelling + first-detection pass covers the
// tiles of all fields of a type in one grid (a global tile index is mapped to
// its field by binary search over per-field prefix counts), and all sweeps of
// all fields, of both types, run in one cooperative launch (sweep_multi.cuh).
// Each field keeps its own scratch, sweep index and stop state, so its result
// is bit-identical to correcting it alone (pmsz_correct_f32 /
// pmsz_correct_f64).  The same kernels serve the continuous-batching server
// (server.cu), where fields join and leave between sweeps.
#include "batch.h"
#include "sweep_multi.cuh"

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

namespace pmsz {

template <typename T>
__global__ void __launch_bounds__(kThreads, 5) k_first_multi(const Inst<T> *__restrict__ inst,
                                                            const uint32_t *__restrict__ tpre, int n) {
    extern __shared__ __align__(128) unsigned char march_smem[];
    CopyMarch<T, kFirst> &sm = *reinterpret_cast<CopyMarch<T, kFirst> *>(march_smem);
    const int i = find_seg(tpre, n, blockIdx.x);
    const Inst<T> &I = inst[i];
    const uint32_t lt = blockIdx.x - __ldg(tpre + i);
    const uint32_t bx = lt % I.tiles_x, rest = lt / I.tiles_x;
    const uint32_t by = rest % I.tiles_y, bz = rest / I.tiles_y;
    const MarchArgs<T> a{I.f, I.fh, I.codes, I.hp, I.req, I.act1, I.slots, I.freq, I.f1};
    const int x = static_cast<int>(bx), y = static_cast<int>(by), z = static_cast<int>(bz);
    if (march_inside(I.g, x, y, z))
        march_copies<T, kFirst, false>(sm, a, I.g, x, y, z);
    else
        march_copies<T, kFirst, true>(sm, a, I.g, x, y, z);
}
template <typename T>
int launch_first_multi(const Inst<T> *inst, const uint32_t *tpre, int n, uint32_t tiles, cudaStream_t s) {
    PMSZ_CUDA(allow_smem(k_first_multi<T>, sizeof(CopyMarch<T, kFirst>)));
    k_first_multi<T><<<tiles, dim3(kTX, kThreads / kTX, 1), sizeof(CopyMarch<T, kFirst>), s>>>(inst, tpre, n);
    PMSZ_CUDA(cudaGetLastError());
    return PMSZ_OK;
}
template int launch_first_multi<float>(const Inst<float> *, const uint32_t *, int, uint32_t, cudaStream_t);
template int launch_first_multi<double>(const Inst<double> *, const uint32_t *, int, uint32_t, cudaStream_t);

int launch_multi_sweeps(const MultiSweeps &a, cudaStream_t s) {
    static std::mutex mu;
    static std::vector<unsigned> known;  // resident blocks per device
    unsigned blocks = 0;
    {
        int dev = 0;
        PMSZ_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        if (static_cast<size_t>(dev) >= known.size()) known.resize(static_cast<size_t>(dev) + 1, 0u);
        if (!known[static_cast<size_t>(dev)]) {
            int sms = 0, per_sm = 0, coop = 0;
            PMSZ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            PMSZ_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
            if (!coop) return set_error(PMSZ_ERR_CUDA, "device does not support cooperative launches");
            PMSZ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweeps_multi, kSweepBlock, 0));
            if (per_sm < 1) return set_error(PMSZ_ERR_CUDA, "sweep kernel does not fit on an SM");
            known[static_cast<size_t>(dev)] = static_cast<unsigned>(per_sm * sms);
        }
        blocks = known[static_cast<size_t>(dev)];
    }
    const uint64_t groups = 8ull * std::max(a.t32.chunks, a.t64.chunks);
    const unsigned grid = static_cast<unsigned>(
        std::max<uint64_t>(1, std::min<uint64_t>((groups + kSweepWarps - 1) / kSweepWarps, blocks)));
    MultiSweeps copy = a;
    void *args[] = {&copy};
    PMSZ_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_sweeps_multi), dim3(grid), dim3(kSweepBlock),
                                          args, 0, s));
    return PMSZ_OK;
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
template <typename T>
int MultiRun<T>::setup(const std::vector<FieldSpec<T>> &specs, int64_t max_sweeps_, int q) {
    n = static_cast<int>(specs.size());
    max_sweeps = max_sweeps_;
    if (n < 1 || n > kMaxBatch) return set_error(PMSZ_ERR_ARG, "batch size must be in 1..4096");
    host.assign(n, Inst<T>{});
    tpre.assign(n + 1, 0);
    cpre.assign(n + 1, 0);
    std::vector<size_t> o_zero(n), o_rest(n);
    std::vector<FieldScratch> fs;
    size_t zero_bytes = 0, rest_bytes = 0;
    uint64_t tiles = 0, chunks = 0, columns = 0;
    voxels = 0;
    for (const FieldSpec<T> &sp : specs) {
        voxels += sp.nx * sp.ny * sp.nz;
        columns += column_planes(sp.nx, sp.ny, sp.nz);
    }
    const int zc = batch_depth(voxels, n, sizeof(T), columns);  // one first-pass launch covers the batch
    for (int i = 0; i < n; ++i) {
        Geom g = make_geom(specs[i].nx, specs[i].ny, specs[i].nz);
        g.zc = zc;
        fs.emplace_back(g, sizeof(T));
        o_zero[i] = zero_bytes;
        o_rest[i] = rest_bytes;
        zero_bytes += fs[i].zero;
        rest_bytes += fs[i].total - fs[i].zero;
        Inst<T> &I = host[i];
        I.f = specs[i].f;
        I.fh = specs[i].fh;
        I.g = g;
        I.eps = static_cast<T>(specs[i].eb);
        I.delta = static_cast<T>(specs[i].eb / static_cast<double>(q));  // pMSz.cu:2814
        I.q = q;
        I.max_sweeps = max_sweeps;
        I.active = 1;
        I.first = 1;
        I.stride = n;
        I.tiles_x = static_cast<uint32_t>(g.wpr);
        I.tiles_y = static_cast<uint32_t>((g.ny + kMY - 1) / kMY);
        tpre[i] = static_cast<uint32_t>(tiles);
        cpre[i] = static_cast<uint32_t>(chunks);
        tiles += static_cast<uint64_t>(I.tiles_x) * I.tiles_y * static_cast<uint64_t>((g.nz + g.zc - 1) / g.zc);
        chunks += sweep_chunks(g);
        if (tiles >= (1ull << 31) || chunks >= (1ull << 31)) return set_error(PMSZ_ERR_ARG, "batch too large");
    }
    tpre[n] = static_cast<uint32_t>(tiles);
    cpre[n] = static_cast<uint32_t>(chunks);
    const size_t slot_bytes = sizeof(SweepSlot) * static_cast<size_t>(max_sweeps) * n;
    const size_t o_z = ws.reserve<unsigned char>(zero_bytes + slot_bytes);
    const size_t o_other = ws.reserve<unsigned char>(rest_bytes);
    const size_t o_inst = ws.reserve<Inst<T>>(n);
    const size_t o_pre = ws.reserve<uint32_t>(2 * (n + 1));
    const size_t o_ctl = ws.reserve<SweepCtl>(1);
    const int rc = ws.commit();
    if (rc) return rc;
    zero_base = ws.at<unsigned char>(o_z);
    zero_total = zero_bytes + slot_bytes;
    slots = reinterpret_cast<SweepSlot *>(zero_base + zero_bytes);
    for (int i = 0; i < n; ++i) {
        fs[i].point(host[i], zero_base + o_zero[i], ws.at<unsigned char>(o_other) + o_rest[i] - fs[i].zero);
        host[i].slots = slots + i;
    }
    dinst = ws.at<Inst<T>>(o_inst);
    dtpre = ws.at<uint32_t>(o_pre);
    dcpre = dtpre + (n + 1);
    ctl = ws.at<SweepCtl>(o_ctl);
    PMSZ_CUDA(cudaMemsetAsync(zero_base, 0, zero_total, s));
    return PMSZ_OK;
}

template <typename T>
int MultiRun<T>::upload() {  // (from pageable memory: the copies are done with it when they return)
    PMSZ_CUDA(cudaMemcpyAsync(dinst, host.data(), host.size() * sizeof(Inst<T>), cudaMemcpyHostToDevice, s));
    std::vector<uint32_t> pre(tpre);
    pre.insert(pre.end(), cpre.begin(), cpre.end());
    PMSZ_CUDA(cudaMemcpyAsync(dtpre, pre.data(), pre.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
    return PMSZ_OK;
}

template <typename T>
int MultiRun<T>::start() {
    const int rc = upload();
    if (rc) return rc;
    return launch_first_multi<T>(dinst, dtpre, n, tpre[n], s);
}

template <typename T>
SweepTable<T> MultiRun<T>::table() const {
    SweepTable<T> t;
    t.inst = dinst;
    t.cpre = dcpre;
    t.n = n;
    t.chunks = cpre[n];
    return t;
}

template <typename T>
int MultiRun<T>::set_zchunk(int zc) {
    uint64_t tiles = 0;
    zc = march_depth(zc);
    for (int i = 0; i < n; ++i) {
        Inst<T> &I = host[i];
        I.g.zc = zc;
        tpre[i] = static_cast<uint32_t>(tiles);
        tiles += static_cast<uint64_t>(I.tiles_x) * I.tiles_y * static_cast<uint64_t>((I.g.nz + zc - 1) / zc);
        if (tiles >= (1ull << 31)) return set_error(PMSZ_ERR_ARG, "batch too large");
    }
    tpre[n] = static_cast<uint32_t>(tiles);
    return PMSZ_OK;
}

template <typename T>
int MultiRun<T>::tune_zchunk() {
    int m = 0, maxnz = 1;
    const int *cands = zchunk_candidates(&m);
    uint64_t columns = 0;
    for (const Inst<T> &I : host) {
        maxnz = std::max(maxnz, I.g.nz);
        columns += column_planes(static_cast<size_t>(I.g.nx), static_cast<size_t>(I.g.ny), static_cast<size_t>(I.g.nz));
    }
    EventTimer et;
    int rc = et.init();
    if (rc) return rc;
    auto time = [&](int zc, float &t_best) -> int {  // best of two after a warm-up
        if ((rc = set_zchunk(zc)) || (rc = upload())) return rc;
        t_best = 0.f;
        for (int rep = 0; rep < 3; ++rep) {
            PMSZ_CUDA(cudaMemsetAsync(zero_base, 0, zero_total, s));
            PMSZ_CUDA(cudaEventRecord(et.ev[0], s));
            if ((rc = launch_first_multi<T>(dinst, dtpre, n, tpre[n], s))) return rc;
            PMSZ_CUDA(cudaEventRecord(et.ev[1], s));
            PMSZ_CUDA(cudaEventSynchronize(et.ev[1]));
            float t = 0.f;
            PMSZ_CUDA(cudaEventElapsedTime(&t, et.ev[0], et.ev[1]));
            if (rep > 0 && (t_best == 0.f || t < t_best)) t_best = t;
        }
        return PMSZ_OK;
    };
    int best = cands[0];
    float best_ms = 0.f, t = 0.f;
    for (int c = 0; c < m; ++c) {
        if ((rc = time(cands[c], t))) return rc;
        if (c == 0 || t < best_ms) {
            best_ms = t;
            best = cands[c];
        }
        if (cands[c] >= maxnz) break;  // deeper columns are one chunk for every field
    }
    // and the depth by size, where it is none of them (as autotune_impl)
    const int own = default_depth(columns);
    bool by_size = false;
    if (own < cands[0]) {
        if ((rc = time(own, t))) return rc;
        by_size = t <= best_ms;
    }
    record_batch_zchunk(voxels, n, sizeof(T), best, by_size);
    if (by_size) best = own;
    if ((rc = set_zchunk(best))) return rc;
    PMSZ_CUDA(cudaMemsetAsync(zero_base, 0, zero_total, s));
    return PMSZ_OK;
}

template struct MultiRun<float>;
template struct MultiRun<double>;

// The sweeps of the runs that are set up (either may be null) and their logs.
// The first log rows come back with the sweep count; the statuses are rebuilt
// from the slot rows with the stop rule that the device applied.
static int run_batch(MultiRun<float> *r32, MultiRun<double> *r64, std::vector<BatchOutcome> &o32,
                     std::vector<BatchOutcome> &o64, cudaStream_t s) {
    int rc;
    if (r32 && (rc = r32->start())) return rc;
    if (r64 && (rc = r64->start())) return rc;
    MultiSweeps a;
    if (r32) a.t32 = r32->table();
    if (r64) a.t64 = r64->table();
    a.ctl = r32 ? r32->ctl : r64->ctl;
    PMSZ_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(SweepCtl), s));
    if ((rc = launch_multi_sweeps(a, s))) return rc;
    // the sweep count and, up to 256 KB a type, the first rows in pinned memory
    auto ahead = [](int n, int64_t max_sweeps) {
        return static_cast<int64_t>(std::min<size_t>(static_cast<size_t>(max_sweeps), (256u << 10) / (sizeof(SweepSlot) * n)));
    };
    const int64_t p32 = r32 ? ahead(r32->n, r32->max_sweeps) : 0, p64 = r64 ? ahead(r64->n, r64->max_sweeps) : 0;
    const size_t b32 = r32 ? sizeof(SweepSlot) * static_cast<size_t>(p32) * r32->n : 0,
                 b64 = r64 ? sizeof(SweepSlot) * static_cast<size_t>(p64) * r64->n : 0;
    unsigned char *hb = static_cast<unsigned char *>(host_pinned(256 + b32 + b64));
    if (!hb) return set_error(PMSZ_ERR_OOM, "pinned host allocation failed");
    PMSZ_CUDA(cudaMemcpyAsync(hb, a.ctl, sizeof(SweepCtl), cudaMemcpyDeviceToHost, s));
    if (b32) PMSZ_CUDA(cudaMemcpyAsync(hb + 256, r32->slots, b32, cudaMemcpyDeviceToHost, s));
    if (b64) PMSZ_CUDA(cudaMemcpyAsync(hb + 256 + b32, r64->slots, b64, cudaMemcpyDeviceToHost, s));
    PMSZ_CUDA(cudaStreamSynchronize(s));
    if (reinterpret_cast<const SweepCtl *>(hb)->err) return set_error(PMSZ_ERR_CUDA, kBarrierMissing);
    const int64_t total = reinterpret_cast<const SweepCtl *>(hb)->iters;  // sweeps 0 .. total - 1
    auto collect = [&](auto *run, const unsigned char *head, int64_t have, std::vector<BatchOutcome> &out) -> int {
        if (!run) return PMSZ_OK;
        const int n = run->n;
        const int64_t rows = std::min(total, run->max_sweeps);
        std::vector<SweepSlot> more;
        if (rows > have) {
            more.resize(static_cast<size_t>(rows - have) * n);
            PMSZ_CUDA(cudaMemcpyAsync(more.data(), run->slots + have * n, more.size() * sizeof(SweepSlot),
                                      cudaMemcpyDeviceToHost, s));
            PMSZ_CUDA(cudaStreamSynchronize(s));
        }
        const SweepSlot *first = reinterpret_cast<const SweepSlot *>(head);
        out.assign(n, BatchOutcome{});
        for (int i = 0; i < n; ++i) {
            BatchOutcome &o = out[i];
            for (int64_t k = 0; k < rows; ++k) {
                const SweepSlot &h = k < have ? first[k * n + i] : more[static_cast<size_t>(k - have) * n + i];
                o.log.push_back(h);
                if (k == 0 && h.bad) {
                    o.status = PMSZ_ERR_ARG;
                    o.message = "input contains NaN or the value 1e30 (the reference's halo sentinel)";
                    break;
                }
                if (sweep_stops(h.fmax, h.fmin, h.fdir, h.progressed, k + 1, run->max_sweeps)) break;
            }
            if (o.status == PMSZ_ERR_ARG) continue;
            const SweepSlot &last = o.log.back();
            if (last.fmax == 0 && last.fmin == 0 && last.fdir == 0) {
                o.status = PMSZ_OK;
            } else {
                o.status = PMSZ_ERR_NOT_CONVERGED;
                o.message = last.progressed == 0
                                ? "a sweep requested edits that changed nothing (all requested vertices clamped)"
                                : "max_sweeps reached before convergence";
            }
        }
        return PMSZ_OK;
    };
    if ((rc = collect(r32, hb + 256, p32, o32))) return rc;
    return collect(r64, hb + 256 + b32, p64, o64);
}

// Tunes (where asked to) and sets one type's run up.
template <typename T>
static int prepare_run(MultiRun<T> &run, const std::vector<FieldSpec<T>> &specs, const pmsz_opts *opts, cudaStream_t s) {
    const int q = opts ? opts->q : 5;
    const int64_t max_sweeps = opts && opts->max_sweeps > 0 ? opts->max_sweeps : 10000;
    if (q < 1 || q > 255) return set_error(PMSZ_ERR_ARG, "q must be in 1..255");
    int rc = PMSZ_OK;
    const bool tune = opts && (opts->flags & PMSZ_FLAG_AUTOTUNE);
    if (tune)  // the first field of each untuned shape class tunes it (its single-call parameters)
        for (const FieldSpec<T> &sp : specs)
            if (!tune_known(sp.nx, sp.ny, sp.nz, sizeof(T)) &&
                (rc = autotune_impl<T>(sp.f, sp.fh, sp.nx, sp.ny, sp.nz, nullptr, s)))
                return rc;
    if ((rc = run.setup(specs, max_sweeps, q))) return rc;
    if (tune && !batch_tune_known(run.voxels, run.n, sizeof(T)) && (rc = run.tune_zchunk())) return rc;
    return PMSZ_OK;
}

// Both types together; one after the other where their scratch does not fit at
// once.
static int batch_impl(const std::vector<FieldSpec<float>> &f32, const std::vector<FieldSpec<double>> &f64,
                      const pmsz_opts *opts, std::vector<BatchOutcome> &o32, std::vector<BatchOutcome> &o64,
                      cudaStream_t s) {
    int rc = PMSZ_OK;
    std::unique_ptr<MultiRun<float>> r32;
    std::unique_ptr<MultiRun<double>> r64;
    if (!f32.empty()) {
        r32 = std::make_unique<MultiRun<float>>(s);
        if ((rc = prepare_run(*r32, f32, opts, s))) return rc;
    }
    if (!f64.empty()) {
        r64 = std::make_unique<MultiRun<double>>(s);
        rc = prepare_run(*r64, f64, opts, s);
        if (rc == PMSZ_ERR_OOM && r32) {
            r64.reset();
            if ((rc = run_batch(r32.get(), nullptr, o32, o64, s))) return rc;
            r32.reset();
            r64 = std::make_unique<MultiRun<double>>(s);
            rc = prepare_run(*r64, f64, opts, s);
        }
        if (rc) return rc;
    }
    if ((rc = run_batch(r32.get(), r64.get(), o32, o64, s))) return rc;
    if (r32 && (rc = r32->ws.release())) return rc;
    return r64 ? r64->ws.release() : PMSZ_OK;
}

static void fill_result(const BatchOutcome &o, pmsz_result *res) {
    if (!res) return;
    res->sweeps = static_cast<int64_t>(o.log.size());
    res->iteration = res->sweeps + 1;
    uint64_t e = 0;
    for (const SweepSlot &h : o.log) e += h.requested;
    res->edits = e;
    if (res->sweep_log && res->sweep_log_cap > 0) {
        const size_t m = std::min<size_t>(o.log.size(), static_cast<size_t>(res->sweep_log_cap));
        std::memcpy(res->sweep_log, o.log.data(), m * sizeof(SweepSlot));
    }
    res->ms_first_pass = res->ms_detect = res->ms_apply = res->ms_total = 0.0;
    res->launches = 0;
}

int correct_batch(const pmsz_field *fields, int count, const pmsz_opts *opts, pmsz_result *results, int *statuses,
                  cudaStream_t s) {
    if (!fields || count < 1) return set_error(PMSZ_ERR_ARG, "empty batch");
    std::vector<int> st(count, PMSZ_OK);
    std::vector<FieldSpec<float>> f32;
    std::vector<FieldSpec<double>> f64;
    std::vector<int> i32, i64;
    for (int i = 0; i < count; ++i) {
        const pmsz_field &F = fields[i];
        int rc = check_geom(F.nx, F.ny, F.nz);
        if (!rc && (!F.f || !F.fhat)) rc = set_error(PMSZ_ERR_ARG, "null field pointer");
        if (!rc && (!(F.eb > 0.0) || !(F.eb < 1e300))) rc = set_error(PMSZ_ERR_ARG, "error bound must be positive and finite");
        if (!rc && F.elem_size != 4 && F.elem_size != 8) rc = set_error(PMSZ_ERR_ARG, "elem_size must be 4 or 8");
        if (rc) {
            st[i] = rc;
            continue;
        }
        if (F.elem_size == 4) {
            f32.push_back({static_cast<const float *>(F.f), static_cast<float *>(F.fhat), F.nx, F.ny, F.nz, F.eb});
            i32.push_back(i);
        } else {
            f64.push_back({static_cast<const double *>(F.f), static_cast<double *>(F.fhat), F.nx, F.ny, F.nz, F.eb});
            i64.push_back(i);
        }
    }
    std::vector<BatchOutcome> o32, o64;
    if (!f32.empty() || !f64.empty()) {
        const int rc = batch_impl(f32, f64, opts, o32, o64, s);
        if (rc) return rc;
    }
    for (size_t j = 0; j < i32.size(); ++j) {
        st[i32[j]] = o32[j].status;
        fill_result(o32[j], results ? results + i32[j] : nullptr);
    }
    for (size_t j = 0; j < i64.size(); ++j) {
        st[i64[j]] = o64[j].status;
        fill_result(o64[j], results ? results + i64[j] : nullptr);
    }
    int worst = PMSZ_OK;
    for (int i = 0; i < count; ++i) {
        if (statuses) statuses[i] = st[i];
        if (st[i] != PMSZ_OK && worst == PMSZ_OK) worst = st[i];
    }
    for (const auto *o : {&o32, &o64})
        for (const BatchOutcome &b : *o)
            if (b.status != PMSZ_OK && !b.message.empty()) set_error(b.status, b.message);
    return worst;
}

}  // namespace pmsz

using namespace pmsz;

extern "C" int pmsz_correct_batch(const pmsz_field *fields, int count, const pmsz_opts *opts, pmsz_result *results,
                                  int *statuses, void *stream) {
    return guarded([&] { return correct_batch(fields, count, opts, results, statuses, as_stream(stream)); });
}
