// The transport's host code (k_transport.cu) over a stand-in CUDA runtime.
#include "fake_cuda.h"
#include "k_transport.cu"

namespace scf_mem {
std::atomic<long long> fail_countdown{0}, live{0};
}

extern "C" void scenario(const char *)
{
    scf_clsvof_ctx *ctx = nullptr;
    const int rc = scf_clsvof_create(&ctx, 6, 5, 4, 0);
    std::printf("%d %d\n", rc, fake::left(nullptr));
    std::fflush(stdout);
}
