// Device time of the BiCGStab sums over a grid of many blocks (k_bicgstab.cu),
// us per launch.
#include <vector>

#include "k_bicgstab.cu"

namespace pred {
namespace {
template <int KIND>
float us_per_sum(const Red &R, int nb, cudaStream_t st)
{
    constexpr int REPS = 200;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    for (int q = 0; q < 20; ++q) sum_blocks<KIND>(R, nb, st);
    cudaEventRecord(a, st);
    for (int q = 0; q < REPS; ++q) sum_blocks<KIND>(R, nb, st);
    cudaEventRecord(b, st);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return ms * 1e3f / REPS;
}
}  // namespace
}  // namespace pred

// us[0..2]: r0.v; t.s and t.t; r0.r and r.r.  Nothing converges or breaks down:
// every partial is 1.
extern "C" int sum_cost(int nb, float *us)
{
    using namespace pred;
    std::vector<double> ones(4 * (size_t)nb, 1.0);
    BcgScalars h{};
    h.rho = h.alpha = h.omega = 1.0;
    h.target = -1.0;
    Red R{};
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    cudaMalloc(&R.partials, ones.size() * sizeof(double));
    cudaMalloc(&R.sc, sizeof(h));
    cudaMemcpy(R.partials, ones.data(), ones.size() * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(R.sc, &h, sizeof(h), cudaMemcpyHostToDevice);
    cudaDeviceSynchronize();
    us[0] = us_per_sum<BR_ALPHA>(R, nb, st);
    us[1] = us_per_sum<BR_OMEGA>(R, nb, st);
    us[2] = us_per_sum<BR_RHO>(R, nb, st);
    cudaMemcpy(&h, R.sc, sizeof(h), cudaMemcpyDeviceToHost);
    const int rc = (int)cudaGetLastError();
    cudaFree(R.partials);
    cudaFree(R.sc);
    cudaStreamDestroy(st);
    return rc ? rc : h.done ? -1 : h.rr == (double)nb ? 0 : -2;
}
