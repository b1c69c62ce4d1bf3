// server.cu -- continuous-batching correction server (pmsz_server_*).
//
// The reference corrects one field per program run.  The server takes
// correction jobs from any host thread and runs them on one GPU with
// continuous batching: a worker thread repeats generations, and in each one
//   1. admits queued jobs in arrival order while the HBM budget (the job's
//      two fields plus its scratch) and the job-slot limit allow,
//   2. runs the fused first pass of the jobs admitted now, then sweeps of all
//      running jobs of both types in one cooperative launch (the multi-field
//      kernels of batch.cu), which ends after the sweep at which some job has
//      stopped or a new job was submitted,
//   3. reads where each job stands and retires finished jobs (waiters woken,
//      scratch freed).
// A job that arrives while others run joins at the next sweep, so its work
// overlaps theirs on the device.  Every job keeps its own scratch, sweep index
// and stop state: its corrected field is bit-identical to running it alone
// through pmsz_correct_*.
//
// A generation used to be one sweep, with up to nine launches, two copies and a
// read-back for each type: a burst of 24 mixed jobs (18 million voxels) took
// 8.6 ms, now 3.6.  What is left is the depth of the longest job's sweeps and a
// generation's fixed costs for every job that ends.
#include "batch.h"

#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <memory>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <vector>

namespace pmsz {

using Clock = std::chrono::steady_clock;

struct Job {
    uint64_t id = 0;
    pmsz_field fd{};
    Geom g{};
    size_t bytes = 0;      // budget charge: fields + scratch
    unsigned char *scratch = nullptr;
    size_t scratch_bytes = 0;
    int64_t k = 0;
    bool first = true;
    bool over = false;     // the worker's: no sweep left (done follows when the job is retired)
    bool done = false;     // under the server's lock: its waiters may release it
    int status = PMSZ_ERR_NOT_CONVERGED;
    int64_t sweeps = 0;
    uint64_t edits = 0;
    Clock::time_point t_submit, t_start, t_done;
};

// A job's scratch: the zeroed part of FieldScratch, its sweep slots (zeroed
// too), then the rest.
static size_t slot_bytes(int64_t max_sweeps) {
    return (sizeof(SweepSlot) * static_cast<size_t>(max_sweeps) + 255) & ~static_cast<size_t>(255);
}

template <typename T>
static Inst<T> make_inst(const Job &j, int q, int64_t max_sweeps) {
    Inst<T> I{};
    const Geom &g = j.g;
    const FieldScratch fs(g, sizeof(T));
    fs.point(I, j.scratch, j.scratch + slot_bytes(max_sweeps));
    I.slots = reinterpret_cast<SweepSlot *>(j.scratch + fs.zero);
    I.f = static_cast<const T *>(j.fd.f);
    I.fh = static_cast<T *>(j.fd.fhat);
    I.stride = 1;
    I.g = g;
    I.eps = static_cast<T>(j.fd.eb);
    I.delta = static_cast<T>(j.fd.eb / static_cast<double>(q));
    I.q = q;
    I.max_sweeps = max_sweeps;
    I.k = j.k;
    I.active = 1;
    I.first = j.first ? 1 : 0;
    I.tiles_x = static_cast<uint32_t>(g.wpr);
    I.tiles_y = static_cast<uint32_t>((g.ny + kMY - 1) / kMY);
    return I;
}

class Server {
public:
    explicit Server(const pmsz_server_config &c) : cfg_(c) {
        if (cfg_.max_jobs <= 0 || cfg_.max_jobs > kMaxBatch) cfg_.max_jobs = 256;
        if (cfg_.q <= 0) cfg_.q = 5;
        if (cfg_.max_sweeps <= 0) cfg_.max_sweeps = 10000;
    }
    ~Server() { shutdown(); }

    int start() {
        PMSZ_CUDA(cudaGetDevice(&device_));
        worker_ = std::thread([this] { run(); });
        return PMSZ_OK;
    }

    void shutdown() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (stopping_) return;
            stopping_ = true;
        }
        cv_work_.notify_all();
        if (worker_.joinable()) worker_.join();
    }

    int submit(const pmsz_field &fd, uint64_t *id) {
        int rc = check_geom(fd.nx, fd.ny, fd.nz);
        if (rc) return rc;
        if (!fd.f || !fd.fhat) return set_error(PMSZ_ERR_ARG, "null field pointer");
        if (!(fd.eb > 0.0) || !(fd.eb < 1e300)) return set_error(PMSZ_ERR_ARG, "error bound must be positive and finite");
        if (fd.elem_size != 4 && fd.elem_size != 8) return set_error(PMSZ_ERR_ARG, "elem_size must be 4 or 8");
        auto j = std::make_unique<Job>();
        j->fd = fd;
        j->g = make_geom(fd.nx, fd.ny, fd.nz);
        j->g.zc = first_depth(fd.nx, fd.ny, fd.nz, fd.elem_size);
        j->scratch_bytes = FieldScratch(j->g, fd.elem_size).total + slot_bytes(cfg_.max_sweeps);
        // its fields, its scratch, and 16 bytes a voxel for what the running
        // set shares (a charge that budgets are sized by: more than is held now)
        j->bytes = field_scratch_bytes(j->g, cfg_.max_sweeps) + 2 * j->g.n * fd.elem_size + 2 * sizeof(uint64_t) * j->g.n;
        if (cfg_.hbm_budget_bytes && j->bytes > cfg_.hbm_budget_bytes)
            return set_error(PMSZ_ERR_OOM, "job larger than the server's HBM budget");
        j->t_submit = Clock::now();
        std::lock_guard<std::mutex> lk(mu_);
        if (stopping_) return set_error(PMSZ_ERR_ARG, "server is shutting down");
        if (broken_) return set_error(PMSZ_ERR_CUDA, "the server's worker could not start");
        j->id = ++next_id_;
        *id = j->id;
        pending_.push_back(j.get());
        jobs_[j->id] = std::move(j);
        if (yield_) __atomic_store_n(yield_, 1, __ATOMIC_RELEASE);  // the running launch ends after its sweep
        cv_work_.notify_all();
        return PMSZ_OK;
    }

    int info(uint64_t id, pmsz_job_info *out, double timeout_s) {
        std::unique_lock<std::mutex> lk(mu_);
        auto it = jobs_.find(id);
        if (it == jobs_.end()) return set_error(PMSZ_ERR_ARG, "unknown job id");
        Job *j = it->second.get();
        if (timeout_s != 0.0) {
            auto pred = [&] { return j->done; };
            if (timeout_s < 0) cv_done_.wait(lk, pred);
            else cv_done_.wait_for(lk, std::chrono::duration<double>(timeout_s), pred);
        }
        std::memset(out, 0, sizeof(*out));
        out->done = j->done ? 1 : 0;
        if (!j->done) return PMSZ_OK;
        out->status = j->status;
        out->sweeps = j->sweeps;
        out->edits = j->edits;
        out->queue_ms = std::chrono::duration<double, std::milli>(j->t_start - j->t_submit).count();
        out->run_ms = std::chrono::duration<double, std::milli>(j->t_done - j->t_start).count();
        out->latency_ms = std::chrono::duration<double, std::milli>(j->t_done - j->t_submit).count();
        return PMSZ_OK;
    }

    int release(uint64_t id) {
        std::lock_guard<std::mutex> lk(mu_);
        auto it = jobs_.find(id);
        if (it == jobs_.end() || !it->second->done) return set_error(PMSZ_ERR_ARG, "job unknown or not finished");
        jobs_.erase(it);
        return PMSZ_OK;
    }

private:
    // The running jobs of one type, and where a generation's upload holds them.
    template <typename T>
    struct Group {
        std::vector<Job *> jobs;
        size_t inst = 0, tpre = 0, cpre = 0, report = 0;  // offsets
        uint32_t tiles = 0, chunks = 0;
    };
    // One upload (tables and prefixes of both types) and one read-back
    // (reports) a generation, through buffers that grow to the largest set.
    struct Buffers {
        unsigned char *up = nullptr, *dup = nullptr;    // pinned, device
        unsigned char *rep = nullptr, *drep = nullptr;  // pinned, device: SweepCtl, then the reports
        size_t up_cap = 0, rep_cap = 0;
    };

    static int grow(unsigned char *&host, unsigned char *&dev, size_t &cap, size_t want) {
        if (want <= cap) return PMSZ_OK;
        if (host) cudaFreeHost(host);
        if (dev) cudaFree(dev);
        host = dev = nullptr;
        cap = 0;
        want = std::max<size_t>(2 * want, 64u << 10);
        PMSZ_CUDA(cudaMallocHost(reinterpret_cast<void **>(&host), want));
        PMSZ_CUDA(cudaMalloc(reinterpret_cast<void **>(&dev), want));
        cap = want;
        return PMSZ_OK;
    }

    // Sizes a group's part of the two buffers.
    template <typename T>
    void place(Group<T> &G, size_t &up, size_t &rep) {
        const size_t n = G.jobs.size();
        auto take = [](size_t &at, size_t bytes) {
            const size_t off = at;
            at += (bytes + 255) & ~static_cast<size_t>(255);
            return off;
        };
        G.inst = take(up, n * sizeof(Inst<T>));
        G.tpre = take(up, (n + 1) * sizeof(uint32_t));
        G.cpre = take(up, (n + 1) * sizeof(uint32_t));
        G.report = take(rep, n * sizeof(SweepReport));
    }

    // Writes a group's table and prefixes; tiles are those of the jobs that start now.
    template <typename T>
    int fill(Group<T> &G) {
        const size_t n = G.jobs.size();
        Inst<T> *inst = reinterpret_cast<Inst<T> *>(buf_.up + G.inst);
        uint32_t *tpre = reinterpret_cast<uint32_t *>(buf_.up + G.tpre), *cpre = reinterpret_cast<uint32_t *>(buf_.up + G.cpre);
        uint64_t tiles = 0, chunks = 0;
        for (size_t i = 0; i < n; ++i) {
            const Job &j = *G.jobs[i];
            inst[i] = make_inst<T>(j, cfg_.q, cfg_.max_sweeps);
            tpre[i] = static_cast<uint32_t>(tiles);
            cpre[i] = static_cast<uint32_t>(chunks);
            if (j.first)
                tiles += static_cast<uint64_t>(inst[i].tiles_x) * inst[i].tiles_y * ((j.g.nz + j.g.zc - 1) / j.g.zc);
            chunks += sweep_chunks(j.g);
            if (tiles >= (1ull << 31) || chunks >= (1ull << 31)) return set_error(PMSZ_ERR_ARG, "running set too large");
        }
        tpre[n] = G.tiles = static_cast<uint32_t>(tiles);
        cpre[n] = G.chunks = static_cast<uint32_t>(chunks);
        return PMSZ_OK;
    }

    template <typename T>
    int start_first(const Group<T> &G) {
        if (!G.tiles) return PMSZ_OK;
        return launch_first_multi<T>(reinterpret_cast<const Inst<T> *>(buf_.dup + G.inst),
                                     reinterpret_cast<const uint32_t *>(buf_.dup + G.tpre), static_cast<int>(G.jobs.size()),
                                     G.tiles, s_);
    }

    template <typename T>
    SweepTable<T> table(const Group<T> &G) {
        SweepTable<T> t;
        t.inst = reinterpret_cast<const Inst<T> *>(buf_.dup + G.inst);
        t.cpre = reinterpret_cast<const uint32_t *>(buf_.dup + G.cpre);
        t.n = static_cast<int>(G.jobs.size());
        t.chunks = G.chunks;
        t.report = reinterpret_cast<SweepReport *>(buf_.drep + G.report);
        return t;
    }

    template <typename T>
    void read(const Group<T> &G) {
        const SweepReport *rep = reinterpret_cast<const SweepReport *>(buf_.rep + G.report);
        for (size_t i = 0; i < G.jobs.size(); ++i) {
            Job &j = *G.jobs[i];
            const SweepReport &r = rep[i];
            j.first = false;
            j.k = r.sweeps;
            if (r.running) continue;
            const SweepSlot &h = r.last;
            j.sweeps = r.sweeps;
            j.edits = r.edits;
            j.status = r.sweeps == 1 && h.bad                          ? PMSZ_ERR_ARG
                       : h.fmax == 0 && h.fmin == 0 && h.fdir == 0 ? PMSZ_OK
                                                                   : PMSZ_ERR_NOT_CONVERGED;
            j.over = true;
        }
    }

    // A generation of the running jobs.
    int step(Group<float> &g32, Group<double> &g64) {
        if (g32.jobs.empty() && g64.jobs.empty()) return PMSZ_OK;
        size_t up = 0, rep = 256;
        static_assert(sizeof(SweepCtl) <= 256, "the reports follow the control block");
        place(g32, up, rep);
        place(g64, up, rep);
        int rc;
        if ((rc = grow(buf_.up, buf_.dup, buf_.up_cap, up)) || (rc = grow(buf_.rep, buf_.drep, buf_.rep_cap, rep)) ||
            (rc = fill(g32)) || (rc = fill(g64)))
            return rc;
        PMSZ_CUDA(cudaMemcpyAsync(buf_.dup, buf_.up, up, cudaMemcpyHostToDevice, s_));
        if ((rc = start_first(g32)) || (rc = start_first(g64))) return rc;
        MultiSweeps a;
        if (!g32.jobs.empty()) a.t32 = table(g32);
        if (!g64.jobs.empty()) a.t64 = table(g64);
        a.ctl = reinterpret_cast<SweepCtl *>(buf_.drep);
        a.yield = dyield_;
        a.until_stop = 1;
        PMSZ_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(SweepCtl), s_));
        if ((rc = launch_multi_sweeps(a, s_))) return rc;
        PMSZ_CUDA(cudaMemcpyAsync(buf_.rep, buf_.drep, rep, cudaMemcpyDeviceToHost, s_));
        PMSZ_CUDA(cudaStreamSynchronize(s_));
        if (reinterpret_cast<const SweepCtl *>(buf_.rep)->err) return set_error(PMSZ_ERR_CUDA, kBarrierMissing);
        read(g32);
        read(g64);
        return PMSZ_OK;
    }

    // After a generation that failed: the running jobs end with `rc`, once nothing
    // that it enqueued runs any more, and give back their budget and scratch.
    void fail_running(int rc) {
        cudaStreamSynchronize(s_);
        cudaGetLastError();  // the failed call's: later launches are checked by it
        std::vector<unsigned char *> scratch;
        {
            std::lock_guard<std::mutex> lk(mu_);
            for (Job *j : running_) {
                if (!j->over) j->status = rc;
                if (j->scratch) scratch.push_back(j->scratch);
                j->scratch = nullptr;
                used_ -= j->bytes;
                j->t_done = Clock::now();
                j->done = true;
            }
            running_.clear();
        }
        cv_done_.notify_all();
        for (unsigned char *p : scratch) cudaFreeAsync(p, s_);
    }

    // Where the worker cannot start: nothing will run the jobs.
    void fail_setup(int *flag) {
        cudaGetLastError();
        if (flag) cudaFreeHost(flag);
        if (s_) cudaStreamDestroy(s_);
        s_ = nullptr;
        {
            std::lock_guard<std::mutex> lk(mu_);
            broken_ = true;
            for (Job *j : pending_) {
                j->status = PMSZ_ERR_CUDA;
                j->t_start = j->t_done = Clock::now();
                j->done = true;
            }
            pending_.clear();
        }
        cv_done_.notify_all();
    }

    void run() {
        cudaSetDevice(device_);
        int *flag = nullptr, *dflag = nullptr;
        if (cudaStreamCreateWithFlags(&s_, cudaStreamNonBlocking) != cudaSuccess ||
            cudaHostAlloc(reinterpret_cast<void **>(&flag), sizeof(int), cudaHostAllocMapped) != cudaSuccess ||
            cudaHostGetDevicePointer(reinterpret_cast<void **>(&dflag), flag, 0) != cudaSuccess) {
            fail_setup(flag);
            return;
        }
        *flag = 0;
        dyield_ = dflag;
        {
            std::lock_guard<std::mutex> lk(mu_);
            yield_ = flag;
        }
        retain_pool_once();
        Group<float> g32;
        Group<double> g64;
        while (true) {
            std::vector<Job *> admitted;
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_work_.wait(lk, [&] { return stopping_ || !pending_.empty() || !running_.empty(); });
                if (stopping_ && pending_.empty() && running_.empty()) break;
                __atomic_store_n(yield_, 0, __ATOMIC_RELEASE);  // what is pending is looked at now
                while (!pending_.empty() && static_cast<int>(running_.size() + admitted.size()) < cfg_.max_jobs) {
                    Job *j = pending_.front();
                    if (cfg_.hbm_budget_bytes && used_ + j->bytes > cfg_.hbm_budget_bytes) break;  // FIFO admission
                    pending_.pop_front();
                    used_ += j->bytes;
                    admitted.push_back(j);
                }
            }
            for (Job *j : admitted) {
                j->t_start = Clock::now();
                if (cudaMallocAsync(reinterpret_cast<void **>(&j->scratch), j->scratch_bytes, s_) != cudaSuccess ||
                    cudaMemsetAsync(j->scratch, 0, FieldScratch(j->g, j->fd.elem_size).zero + slot_bytes(cfg_.max_sweeps), s_) != cudaSuccess) {
                    cudaGetLastError();
                    j->status = PMSZ_ERR_OOM;
                    j->over = true;
                }
            }
            {
                std::lock_guard<std::mutex> lk(mu_);
                for (Job *j : admitted) running_.push_back(j);
            }
            g32.jobs.clear();
            g64.jobs.clear();
            for (Job *j : running_)
                if (!j->over) (j->fd.elem_size == 4 ? (std::vector<Job *> &)g32.jobs : g64.jobs).push_back(j);
            if (step(g32, g64) != PMSZ_OK) {
                fail_running(PMSZ_ERR_CUDA);
                continue;
            }
            // retire finished jobs (a waiter may release its job as soon as the lock is free)
            std::vector<Job *> keep;
            std::vector<unsigned char *> done;
            {
                std::lock_guard<std::mutex> lk(mu_);
                for (Job *j : running_) {
                    if (j->over) {
                        if (j->scratch) done.push_back(j->scratch);
                        j->scratch = nullptr;
                        used_ -= j->bytes;
                        j->t_done = Clock::now();
                        j->done = true;
                    } else {
                        keep.push_back(j);
                    }
                }
                running_.swap(keep);
            }
            cv_done_.notify_all();
            for (unsigned char *p : done) cudaFreeAsync(p, s_);
        }
        cudaStreamSynchronize(s_);
        {
            std::lock_guard<std::mutex> lk(mu_);
            yield_ = nullptr;
        }
        cudaFreeHost(flag);
        if (buf_.up) cudaFreeHost(buf_.up);
        if (buf_.dup) cudaFree(buf_.dup);
        if (buf_.rep) cudaFreeHost(buf_.rep);
        if (buf_.drep) cudaFree(buf_.drep);
        buf_ = Buffers{};
        cudaStreamDestroy(s_);
    }

    pmsz_server_config cfg_;
    int device_ = 0;
    cudaStream_t s_ = nullptr;
    Buffers buf_;
    int *yield_ = nullptr;               // mapped: set by a submission (under mu_)
    const volatile int *dyield_ = nullptr;  // its device address
    std::thread worker_;
    std::mutex mu_;
    std::condition_variable cv_work_, cv_done_;
    std::deque<Job *> pending_;
    std::vector<Job *> running_;
    std::unordered_map<uint64_t, std::unique_ptr<Job>> jobs_;
    uint64_t next_id_ = 0;
    size_t used_ = 0;
    bool stopping_ = false;
    bool broken_ = false;  // the worker could not start
};

}  // namespace pmsz

using namespace pmsz;

struct pmsz_server {
    std::unique_ptr<Server> impl;
};

extern "C" int pmsz_server_create(const pmsz_server_config *cfg, pmsz_server **out) {
    return guarded([&] {
        if (!cfg || !out) return set_error(PMSZ_ERR_ARG, "null argument");
        auto s = std::make_unique<pmsz_server>();
        s->impl = std::make_unique<Server>(*cfg);
        const int rc = s->impl->start();
        if (rc) return rc;
        *out = s.release();
        return PMSZ_OK;
    });
}

extern "C" int pmsz_server_submit(pmsz_server *srv, const pmsz_field *field, uint64_t *job_id) {
    return guarded([&] {
        if (!srv || !field || !job_id) return set_error(PMSZ_ERR_ARG, "null argument");
        return srv->impl->submit(*field, job_id);
    });
}

extern "C" int pmsz_server_wait(pmsz_server *srv, uint64_t job_id, double timeout_s, pmsz_job_info *info) {
    return guarded([&] {
        if (!srv || !info) return set_error(PMSZ_ERR_ARG, "null argument");
        return srv->impl->info(job_id, info, timeout_s);
    });
}

extern "C" int pmsz_server_release(pmsz_server *srv, uint64_t job_id) {
    return guarded([&] {
        if (!srv) return set_error(PMSZ_ERR_ARG, "null argument");
        return srv->impl->release(job_id);
    });
}

extern "C" int pmsz_server_destroy(pmsz_server *srv) {
    return guarded([&] {
        if (!srv) return PMSZ_OK;
        srv->impl->shutdown();
        delete srv;
        return PMSZ_OK;
    });
}
