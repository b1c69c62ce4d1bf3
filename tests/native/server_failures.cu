// The correction server (csrc/server.cu) over a fake of the CUDA runtime
// (fake_runtime.cpp) and of the launches it makes, which fail on request; a launch
// of sweeps reports every job as finished.  No GPU is used.  Run as
// server_failures SCENARIO; prints one line per job and the allocations left.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <thread>

#include "../../pmsz_anonymous_gb300/csrc/batch.h"
#include "fake.h"

using namespace fake;

namespace pmsz {
int set_error(int status, const std::string &) { return status; }
int check_geom(size_t, size_t, size_t) { return PMSZ_OK; }
int first_depth(size_t, size_t, size_t, size_t) { return 4; }
void retain_pool_once() {}
template <typename T>
int launch_first_multi(const Inst<T> *, const uint32_t *, int, uint32_t, cudaStream_t) {
    in_flight = true;
    return cudaGetLastError() == cudaSuccess ? PMSZ_OK : PMSZ_ERR_CUDA;  // as a launch is checked
}
template int launch_first_multi<float>(const Inst<float> *, const uint32_t *, int, uint32_t, cudaStream_t);
template int launch_first_multi<double>(const Inst<double> *, const uint32_t *, int, uint32_t, cudaStream_t);
template <typename T>
static void finish(const SweepTable<T> &t) {
    for (int i = 0; i < t.n; ++i) {
        t.report[i] = SweepReport{};
        t.report[i].sweeps = 1;
    }
}
int launch_multi_sweeps(const MultiSweeps &a, cudaStream_t) {
    if (take(fail_sweeps)) return PMSZ_ERR_CUDA;
    finish(a.t32);
    finish(a.t64);
    return PMSZ_OK;
}
}  // namespace pmsz

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "sweeps") fail_sweeps = 1;
    if (what == "buffers") fail_malloc = 1;
    if (what == "scratch") fail_scratch = 1;
    if (what == "setup") fail_host = 1;
    static float f[64], fh[64];
    pmsz_field fd{f, fh, 4, 4, 4, 1e-3, 4, 0};
    const pmsz::Geom g = pmsz::make_geom(4, 4, 4);
    pmsz_server_config cfg{};
    cfg.max_sweeps = 4;
    // room for one job at a time
    cfg.hbm_budget_bytes = pmsz::field_scratch_bytes(g, 4) + 2 * g.n * 4 + 2 * sizeof(uint64_t) * g.n;
    pmsz_server *srv = nullptr;
    if (pmsz_server_create(&cfg, &srv)) return 2;
    for (int k = 0; k < 3; ++k) {
        uint64_t id = 0;
        const int rc = pmsz_server_submit(srv, &fd, &id);
        pmsz_job_info info{};
        if (!rc) pmsz_server_wait(srv, id, 3.0, &info);
        std::printf("job %d submit %d done %d status %d in_flight %d\n", k, rc, info.done, info.done ? info.status : -1,
                    in_flight.load() ? 1 : 0);
        std::fflush(stdout);
        if (!rc && !info.done) std::_Exit(3);  // it would never end
        if (what == "setup") std::this_thread::sleep_for(std::chrono::milliseconds(200));
    }
    pmsz_server_destroy(srv);
    std::printf("left %d\n", live.load());
    return 0;
}
