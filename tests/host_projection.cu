// The projection's host code (scf_api.cu) over a stand-in CUDA runtime, with
// launchers that give work to their stream and form the sums the host waits for.
#include "fake_cuda.h"
#include "scf_kernels.h"

#include <cstdio>
#include <sched.h>

namespace {
double rhs_sum = 4.0, step_sum = 0.0;     // (b, b), and (r, r) after a CG step
std::vector<double> residuals;            // (r, r) of each residual, in order
struct Sum {
    volatile double *box;
    double v;
    bool step;
};
std::vector<Sum> in_flight;               // on their way to the host's memory

// One write becomes visible: writes of different kernels do in any order, here
// a step's sum first, then the oldest.
void land()
{
    for (size_t q = 0; q < in_flight.size(); ++q)
        if (in_flight[q].step) std::swap(in_flight[0], in_flight[q]);
    if (in_flight.empty()) return;
    *in_flight[0].box = in_flight[0].v;
    in_flight.erase(in_flight.begin());
}
void land_all()
{
    while (!in_flight.empty()) land();
}
void mailed(Reducer &R, Mail m, int slot, double v)
{
    R.scal[slot] = v;
    if (R.mail) in_flight.push_back({R.mail + m * MAIL_STRIDE, v, m == MAIL_RR});
}
}  // namespace

extern "C" int sched_yield()
{
    ++fake::yields;
    return 0;
}

void rhs_prologue(const LevelView<double> &, const unsigned char *, double *, bool, Reducer &R, cudaStream_t st, int *)
{
    fake::work("rhs", st);
    mailed(R, MAIL_BB, S_BB, rhs_sum);
}
void final_residual(const LevelView<double> &, const unsigned char *, const double *, const double *, double *, bool,
                    Reducer &R, cudaStream_t st, int *)
{
    fake::work("residual", st);
    const double v = residuals.front();
    residuals.erase(residuals.begin());
    mailed(R, MAIL_RESIDUAL, S_RR, v);
}
template <>
void mg_coarsen<double>(const MgLevel<double> &, MgLevel<double> &, cudaStream_t st, int *) { fake::work("coarsen", st); }
template <>
void mg_coarse_inverse<double>(const MgLevel<double> &, double *, int *, int, bool, cudaStream_t st, int *)
{
    fake::work("inverse", st);
}
template <>
double *mg_vcycle<double>(MgLevel<double> *L, int, const ChebCoef &, const double *, const int *, int, bool, bool,
                          cudaStream_t st, int *, KTimer *, cudaEvent_t ready)
{
    if (ready) cudaStreamWaitEvent(st, ready, 0);
    fake::work("vcycle", st);
    return L[0].xb;
}
template <>
void cg_dot_rz<double>(const LevelView<double> &, const double *, const double *, const double *, Reducer &,
                       cudaStream_t st, int *) { fake::work("dot", st); }
template <>
void cg_pupdate<double>(const LevelView<double> &, const double *, double *, const double *, bool, cudaStream_t st, int *)
{
    fake::work("p", st);
}
void cg_spmv_dot(const LevelView<double> &, const double *, double *, Reducer &, bool, cudaStream_t st, int *, KTimer *)
{
    fake::work("spmv", st);
}
template <>
void cg_update<double>(const LevelView<double> &, double *, double *, const double *, const double *, double *,
                       const LevelView<double> &, double *, double, Reducer &R, cudaStream_t st, int *, KTimer *)
{
    fake::work("update", st);
    mailed(R, MAIL_RR, S_RR, step_sum);
}
cudaError_t coarse_cycle_attr() { return cudaSuccess; }
cudaError_t pair_smem_attr() { return cudaSuccess; }
int smoother_pairs_state() { return 1; }

#include "scf_api.cu"   // after the specialisations

extern "C" void scenario(const char *name)
{
    const std::string what = name;
    fake::on_query = land;
    fake::on_wait = land_all;
    scf_opts o;
    scf_opts_default(&o);
    o.warm_start = what == "warm";
    o.coarse_max_cells = 8;
    scf_ctx *ctx = nullptr;
    if (scf_ctx_create(&ctx, 6, 5, 4, &o) != SCF_OK) return;
    for (int q = 0; q < 6; ++q) ctx->bcp_flag[q] = 0;
    scf_stats st{};
    if (what == "replan") {   // zeroed buffers of a new plan and of the adjoint
        o.coarse_max_cells = 16;
        fake::outstanding.clear();
        const int rc = scf_ctx_set_opts(ctx, &o), rc2 = ensure_adj(ctx);
        std::printf("%d %d %d\n", rc, rc2, fake::left(nullptr));
    }
    if (what == "nonfinite_rhs" || what == "nonfinite_step") {   // what is left when the solve gives up
        (what == "nonfinite_rhs" ? rhs_sum : step_sum) = std::nan("");
        const int rc = solve_impl<double>(ctx, ctx->L64, &st);
        std::printf("%d %d %d\n", rc == SCF_ERR_NONFINITE, fake::left(ctx->st), fake::left(ctx->ist));
    }
    if (what == "zero_rhs") {   // a solve without a V-cycle, then one with: the levels wait for the first inverse
        rhs_sum = 0.0;
        const int rc = solve_impl<double>(ctx, ctx->L64, &st);
        fake::log.clear();
        rhs_sum = 4.0;
        residuals = {0.0};
        const int rc2 = solve_impl<double>(ctx, ctx->L64, &st);
        const std::string joined = "sync " + std::to_string((uintptr_t)ctx->ist);
        size_t wait = fake::log.size(), coarsen = wait;
        for (size_t q = fake::log.size(); q-- > 0;) {
            if (fake::log[q] == joined) wait = q;
            if (fake::log[q].compare(0, 7, "coarsen") == 0) coarsen = q;
        }
        std::printf("%d %d %d\n", rc, rc2, wait < coarsen);
    }
    if (what == "warm") {   // the residual it starts from is not taken for the one it ends with
        ctx->warm_ok = true;
        residuals = {9.0, 0.0, 0.0};
        const int rc = solve_impl<double>(ctx, ctx->L64, &st);
        std::printf("%d %d %g\n", rc, (int)st.rounds, st.rel_residual);
    }
    if (what == "spin" || what == "yield" || what == "block") {   // as the device's flags ask
        fake::device_flags = what == "yield" ? cudaDeviceScheduleYield : what == "block" ? cudaDeviceScheduleBlockingSync
                                                                                         : cudaDeviceScheduleSpin;
        residuals = {0.0};
        fake::waits = 0;
        const int rc = solve_impl<double>(ctx, ctx->L64, &st);
        std::printf("%d %d %d %d\n", rc, fake::queries > 0, fake::yields > 0, fake::waits > 0);
    }
    std::fflush(stdout);
}
