// batch.h -- multi-field correction: the per-field table the multi-field
// kernels read, and the host side shared by pmsz_correct_batch (batch.cu) and
// the continuous-batching server (server.cu).
#pragma once
#include "march.cuh"
#include "internal.h"

#include <string>
#include <vector>

namespace pmsz {

constexpr int kMaxBatch = 4096;

// One field of a multi-field run, as the kernels see it.
template <typename T>
struct Inst {
    const T *f;
    T *fh;
    uint8_t *codes, *cnt;
    uint32_t *hp, *req, *act0, *act1;
    uint8_t *freq, *f0, *f1;  // group flags of req, act0, act1, padded to whole chunks of eight groups
    SweepSlot *slots;   // this field's slot of sweep k is slots[k * stride]
    int64_t stride;
    Geom g;
    T eps, delta;
    int q;
    int64_t max_sweeps;
    int64_t k;          // index of the field's next sweep
    int active;         // runs sweeps
    int first;          // joins now: its fused first pass runs in this generation
    uint32_t tiles_x, tiles_y;
};

template <typename T>
struct FieldSpec {
    const T *f;
    T *fh;
    size_t nx, ny, nz;
    double eb;
};

struct BatchOutcome {
    int status = PMSZ_ERR_NOT_CONVERGED;
    std::string message;
    std::vector<SweepSlot> log;
};

// Scratch of one field, at 256-byte offsets: first what starts at zero
// (counters, bitmaps and their group flags), then codes and, fp64, proxies.  The sweep slots are the caller's.
struct FieldScratch {
    size_t cnt, req, act0, act1, freq, f0, f1, zero, codes, hp, total;
    FieldScratch(const Geom &g, size_t elem) {
        size_t at = 0;
        auto take = [&](size_t bytes) {
            const size_t off = at;
            at += (bytes + 255) & ~static_cast<size_t>(255);
            return off;
        };
        const size_t groups = (g.nwords + kGroupWords - 1) / kGroupWords;
        cnt = take(g.n);
        req = take(4 * g.nwords);
        act0 = take(4 * g.nwords);
        act1 = take(4 * g.nwords);
        freq = take(groups);
        f0 = take(groups);
        f1 = take(groups);
        zero = at;
        codes = take(g.n);
        hp = take(elem == 8 ? 4 * g.n : 0);
        total = at;
    }
    // The table row's scratch pointers: zeroed part at z, the rest at r
    // (r = z where a field's scratch is one piece).
    template <typename T>
    void point(Inst<T> &I, unsigned char *z, unsigned char *r) const {
        I.cnt = z + cnt;
        I.req = reinterpret_cast<uint32_t *>(z + req);
        I.act0 = reinterpret_cast<uint32_t *>(z + act0);
        I.act1 = reinterpret_cast<uint32_t *>(z + act1);
        I.freq = z + freq;
        I.f0 = z + f0;
        I.f1 = z + f1;
        I.codes = r + codes;
        I.hp = sizeof(T) == 8 ? reinterpret_cast<uint32_t *>(r + hp) : nullptr;
    }
};
// Chunks of eight groups (kGroupWords words each) of a field.
inline uint64_t sweep_chunks(const Geom &g) {
    const uint64_t groups = (g.nwords + kGroupWords - 1) / kGroupWords;
    return (groups + 7) / 8;
}

// One type's fields in a k_sweeps_multi launch.
struct SweepReport {
    SweepSlot last;  // of the last sweep run, where the field has stopped
    unsigned long long edits;  // sum of its sweeps' requests, likewise
    long long sweeps;          // run so far
    long long running;
};
template <typename T>
struct SweepTable {
    const Inst<T> *inst = nullptr;
    const uint32_t *cpre = nullptr;  // n + 1 prefixes of sweep_chunks
    int n = 0;
    uint32_t chunks = 0;             // their total
    SweepReport *report = nullptr;   // n, or null: none wanted (a batch reads the slots)
};
struct SweepCtl {  // zero before the launch
    long long iters;  // sweeps run by the launch
    int yield[2];
    uint32_t bar, err;  // the grid barrier's arrivals; kErrBarrier
};
struct MultiSweeps {
    SweepTable<float> t32;
    SweepTable<double> t64;
    SweepCtl *ctl = nullptr;
    const volatile int *yield = nullptr;  // mapped host memory, or null
    int until_stop = 0;                   // end as soon as a field has stopped
};
// The sweeps of both tables: of fields with `first` set from the edits of
// sweep 0 on, of the others from the detection of sweep k on.
int launch_multi_sweeps(const MultiSweeps &a, cudaStream_t s);
// The fused first pass of the fields whose tiles tpre counts (n + 1 prefixes).
template <typename T>
int launch_first_multi(const Inst<T> *inst, const uint32_t *tpre, int n, uint32_t tiles, cudaStream_t s);

// Scratch and table of one batch of same-type fields; slot rows are
// sweep-major (row k holds the slot of sweep k of every field).
template <typename T>
struct MultiRun {
    explicit MultiRun(cudaStream_t st) : s(st), ws(st) {}
    MultiRun(const MultiRun &) = delete;
    MultiRun &operator=(const MultiRun &) = delete;
    int setup(const std::vector<FieldSpec<T>> &specs, int64_t max_sweeps, int q);
    // Uploads the table and the prefixes and launches the first passes.
    int start();
    SweepTable<T> table() const;
    int upload();
    // Sets every field's tile depth (and the tile prefixes) to zc.
    int set_zchunk(int zc);
    // Times the first-pass launch over the whole table at each candidate
    // depth (scratch re-zeroed afterwards), records the fastest for the
    // batch's size class and sets it.
    int tune_zchunk();

    cudaStream_t s;
    Workspace ws;
    int n = 0;
    int64_t max_sweeps = 0;
    std::vector<Inst<T>> host;
    std::vector<uint32_t> tpre, cpre;
    Inst<T> *dinst = nullptr;
    uint32_t *dtpre = nullptr, *dcpre = nullptr;
    SweepCtl *ctl = nullptr;
    SweepSlot *slots = nullptr;
    unsigned char *zero_base = nullptr;  // the scratch that starts zeroed (counters, bitmaps, slots)
    size_t zero_total = 0;
    size_t voxels = 0;
};

// Scratch bytes of one field and its sweep slots, as admission budgets count
// them (codes, counters, proxies, three bitmaps).
inline size_t field_scratch_bytes(const Geom &g, int64_t max_sweeps) {
    auto up = [](size_t b) { return (b + 255) & ~static_cast<size_t>(255); };
    return up(g.n) * 2 + up(4 * g.n) + 3 * up(4 * g.nwords) + up(sizeof(SweepSlot) * static_cast<size_t>(max_sweeps));
}

}  // namespace pmsz
