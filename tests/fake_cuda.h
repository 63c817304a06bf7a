// fake_cuda.h -- a stand-in CUDA runtime for tests of the library's host code
// (linked with -cudart none).  Device memory is host memory.  Work given to a
// stream counts as outstanding until a call waits for that stream; nothing else
// finishes it, so a host path that relies on luck is seen.  The order of the
// calls is kept in fake::log.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace fake {
inline std::map<cudaStream_t, int> outstanding;   // operations per stream; the null stream is the legacy one
inline std::vector<std::string> log;
inline unsigned device_flags = cudaDeviceScheduleAuto;
inline int queries = 0, waits = 0, yields = 0;
inline std::function<void()> on_query, on_wait;   // what lands while the host polls, or waits
inline uintptr_t next = 0x1000;

inline void note(const char *what, cudaStream_t st)
{
    log.push_back(std::string(what) + " " + std::to_string((uintptr_t)st));
}
inline void work(const char *what, cudaStream_t st)
{
    ++outstanding[st];
    note(what, st);
}
inline void wait(const char *what, cudaStream_t st)
{
    if (on_wait) on_wait();
    ++waits;
    outstanding[st] = 0;
    note(what, st);
}
inline int left(cudaStream_t st) { return outstanding[st]; }
inline int left()
{
    int n = 0;
    for (auto &p : outstanding) n += p.second;
    return n;
}
}  // namespace fake
