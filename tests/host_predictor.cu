// The predictor's host code (pred_api.cu) over a stand-in CUDA runtime.
#include "fake_cuda.h"
#include "pred_api.cu"

#include <cstdio>

namespace scf_mem {
std::atomic<long long> fail_countdown{0}, live{0};
}
namespace pred {
int march_len(int, int, int, long long) { return 4; }
dim3 solver_grid(const Dims &) { return dim3(4, 4, 4); }
}

extern "C" void scenario(const char *)
{
    scf_mom_ctx *ctx = nullptr;
    const int rc = scf_mom_create(&ctx, 6, 5, 4, 0);
    std::printf("%d %d\n", rc, fake::left());
    std::fflush(stdout);
}
