// What server_failures.cu asks of fake_runtime.cpp.
#pragma once
#include <atomic>

namespace fake {
extern std::atomic<int> live;  // scratch and device allocations
extern std::atomic<int> fail_malloc, fail_host, fail_scratch, fail_sweeps;  // calls that fail from now on
extern std::atomic<bool> in_flight;  // a first pass was enqueued and not waited for
bool take(std::atomic<int> &n);
}  // namespace fake
