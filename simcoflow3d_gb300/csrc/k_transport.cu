// k_transport.cu -- the CLSVOF interface transport on the device and its C
// ABI (include/scf_clsvof.h).
//
// One time step is six sub-steps; a sub-step is
//   3 x (k_partial_fluxes, k_sweep)  the split sweeps: the geometric fluxes of
//                                  the partly filled cells, gathered into full
//                                  warps, then every cell's update from its
//                                  own two faces (no scatter, no atomics)
//                                  with the divergence term fused in;
//   k_walls                        the wall planes and ghosts;
//   k_normals                      liquid normals and centre distances, and
//                                  the redistancing's resets;
//   k_band_bound, k_band_pairs,    the redistancing over the 9^3 band pairs of
//   k_band_value                   the interface cells, which the last sweep
//                                  has listed: FP32 bounds of every
//                                  pair's distance leave each target its
//                                  least upper bound, then only the pairs
//                                  whose lower bound does not exceed it are
//                                  computed in FP64 and sent with a 64-bit
//                                  atomicMin (non-negative doubles order like
//                                  their bits), so the result is the
//                                  reference's running minimum whatever the
//                                  order.
// The VOF and level set ping-pong through three buffers (the sub-step's
// input, its first sweep's result, which the later sweeps' divergence terms
// read, and the second sweep's result); every sub-step ends in buffer 0.
// The sweeps write interior cells only: k_walls writes the ghost faces into
// all three buffers, and staging fills all three, so their ghosts agree.
// Kernels over cells run on 3-D grids (i along x, j and k as blockIdx.y/z),
// so no thread decodes its cell with integer division.
// Built with -fmad=false: the bodies round like the reference's Fortran.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/scf_clsvof.h"
#include "transport_body.cuh"
#include "scf_launch.cuh"
#include "scf_devmem.h"
#include "scf_stage.h"

using tr::Dims;
using tr::Geo;

struct scf_clsvof_ctx {
    Dims D{};
    int device = 0;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[4] = {};
    std::vector<void *> mem;
    double *geo[6] = {};                 // x, y, z, dx, dy, dz
    double *vf[3] = {}, *ls[3] = {};     // ghosted ping-pong
    double *flo = nullptr, *fhi = nullptr;   // a partial cell's fluxes through its low and high face
    double *dis = nullptr;
    double *nxl = nullptr, *nyl = nullptr, *nzl = nullptr;
    double *fn[3] = {};                  // fluid normals
    double *vel[3] = {};
    double *bc_vel[3] = {};              // W, S, B planes of u, v, w
    double *lvs_bc[6] = {}, *vof_bc[6] = {};
    unsigned long long *key = nullptr;
    uint8_t *fix = nullptr;
    uint8_t *cls = nullptr;              // bit 0: band target, bit 1: level set negative
    unsigned *ub = nullptr;              // least FP32 upper bound of a target's distance (float bits)
    uint32_t *part[2] = {};              // partly filled cells (interior indices) a sweep left, in turn
    unsigned *npart = nullptr;           // how many: one count per sweep of a step
    double *vgeo[3][3] = {};             // U, V, W grid spacings (allocated on first use)
    double *vfld[3][5] = {};             // U, V, W: phiL, nxL, nyL, nzL, vofL
    int lvs_flag[6] = {}, vof_flag[6] = {};
    double lvs_const[6] = {}, vof_const[6] = {};
    double dt = 0.0;
    bool staged = false;
    bool timing = false;
    std::vector<cudaEvent_t> tev;        // 2 per launch of a step when timing
    std::vector<int> tkind;              // kernel kind of each timed launch
    char err[512] = {0};
};

namespace {

constexpr int NT = 256;   // threads per block of the linear kernels
constexpr int NX = 128;   // threads along i of the 3-D kernels

void tr_err(scf_clsvof_ctx *c, const char *fmt, ...)
{
    if (!c) return;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(c->err, sizeof(c->err), fmt, ap);
    va_end(ap);
}

#define TK(call)                                                                            \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess) {                                                            \
            tr_err(ctx, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return e_ == cudaErrorMemoryAllocation ? SCF_ERR_OUT_OF_MEMORY : SCF_ERR_CUDA;   \
        }                                                                                   \
    } while (0)

int blocks_for(size_t n)
{
    const size_t b = (n + NT - 1) / NT;
    return (int)std::min<size_t>(std::max<size_t>(b, 1), (size_t)152 * 64);
}

Geo geo_of(const scf_clsvof_ctx *c)
{
    return Geo{c->geo[0], c->geo[1], c->geo[2], c->geo[3], c->geo[4], c->geo[5]};
}

// ---- kernels -------------------------------------------------------------

// Both reconstruction passes look at every cell for the few the interface
// crosses and then do hundreds of FP64 operations on each of those.  Done
// where they are found, a warp runs all of it for one or two lanes, so a block
// first collects its cells -- RB_X x RB_YZ x RB_YZ of them -- in shared memory
// and then takes them one per thread.
constexpr int RB_X = 128, RB_YZ = 4, RB_CELLS = RB_X * RB_YZ * RB_YZ, RB_THREADS = 256;

struct RbCell {
    int i, j, k;
};
__device__ __forceinline__ RbCell rb_cell(int e)   // cell e of the block
{
    const int r = e / RB_X;
    return RbCell{(int)blockIdx.x * RB_X + e % RB_X + 1, (int)blockIdx.y * RB_YZ + r % RB_YZ + 1,
                  (int)blockIdx.z * RB_YZ + r / RB_YZ + 1};
}
inline dim3 rb_grid(const Dims &D)
{
    return dim3((D.I + RB_X - 1) / RB_X, (D.J + RB_YZ - 1) / RB_YZ, (D.K + RB_YZ - 1) / RB_YZ);
}

// Appends the marked lanes' cells to a list (one atomic per warp; the list's
// order does not matter).  Called by whole warps.
__device__ __forceinline__ void append(bool mark, uint32_t cell, uint32_t *list, unsigned *count)
{
    const unsigned mask = __ballot_sync(0xffffffffu, mark);
    if (!mask) return;
    const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (mark) list[base + __popc(mask & ((1u << lane) - 1u))] = cell;
}

// Interface_Reconstruct of a partly filled cell and the fluxes it sends
// through its faces along the sweep's axis (the only use a sweep has for the
// normals).
__device__ __forceinline__ void flux_cell(const Dims &D, const Geo &G, const tr::SweepIn &S, int i, int j, int k,
                                          double *flo, double *fhi)
{
    double n1, n2, n3, s, fl, fh;
    tr::reconstruct(D, G, S.vfl, S.phi, i, j, k, n1, n2, n3, s);
    tr::partial_fluxes(D, G, S, i, j, k, n1, n2, n3, s, fl, fh);
    const size_t g = D.g(i, j, k);
    flo[g] = fl;
    fhi[g] = fh;
}

// The partial cells' fluxes from the list the sweep before left.  Bound: the
// latency of one cell's chain (some 700 FP64 operations and the branches its
// warp's other cells take), so the cells spread thinly: single-warp blocks,
// and as few cells per warp as give three warps to each SM.
__global__ void __launch_bounds__(32) k_partial_fluxes(const __grid_constant__ Dims D, const __grid_constant__ Geo G,
                                                       const __grid_constant__ tr::SweepIn S, const uint32_t *__restrict__ list,
                                                       const unsigned *__restrict__ count, double *__restrict__ flo,
                                                       double *__restrict__ fhi)
{
    after_previous();
    const unsigned n = *count, per = min(32u, max(4u, (n + 152 * 3 - 1) / (152 * 3)));
    if (threadIdx.x >= per) return;
    for (unsigned long long q = (unsigned long long)blockIdx.x * per + threadIdx.x; q < n;
         q += (unsigned long long)gridDim.x * per) {
        int i, j, k;
        tr::cell_of(D, list[q], i, j, k);
        flux_cell(D, G, S, i, j, k, flo, fhi);
    }
}

// The same for a state no sweep has listed (the first sweep of a call): a
// block looks for its partial cells first.
__global__ void __launch_bounds__(RB_THREADS) k_partial_fluxes_scan(const __grid_constant__ Dims D, const __grid_constant__ Geo G,
                                                                    const __grid_constant__ tr::SweepIn S,
                                                                    double *__restrict__ flo, double *__restrict__ fhi)
{
    after_previous();
    __shared__ unsigned short list[RB_CELLS];
    __shared__ int count;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RB_CELLS / RB_THREADS; ++q) {
        const int e = q * RB_THREADS + threadIdx.x;
        const RbCell c = rb_cell(e);
        if (c.i <= D.I && c.j <= D.J && c.k <= D.K && tr::partial_cell(S.vfl[D.g(c.i, c.j, c.k)]))
            list[atomicAdd(&count, 1)] = (unsigned short)e;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < count; q += RB_THREADS) {
        const RbCell c = rb_cell(list[q]);
        flux_cell(D, G, S, c.i, c.j, c.k, flo, fhi);
    }
}

// The liquid normals and the distances from the cell centres after the sweeps
// (Clsvof_Scheme 767-778) and the redistancing's per-cell state.  The first
// kNormalBlocks blocks take the listed partial cells one per thread, the
// others go over the grid a row each: resets, zero normals away from the
// interface, and the full or empty cells beside the opposite phase, which
// reconstruct too.
constexpr int kNormalBlocks = 152 * 2, NB_THREADS = 128;

struct NormalOut {
    double *nxl, *nyl, *nzl, *dis;
    unsigned long long *key;
    uint8_t *fix, *cls;
    unsigned *ub;
};
__device__ __noinline__ void normal_cell(const Dims &D, const Geo &G, const double *vfl, const double *phi,
                                         const NormalOut &O, int i, int j, int k)
{
    double n1, n2, n3, d1;
    tr::reconstruct(D, G, vfl, phi, i, j, k, n1, n2, n3, d1);
    const size_t g = D.g(i, j, k), t = D.n(i, j, k);
    O.nxl[g] = n1;
    O.nyl[g] = n2;
    O.nzl[g] = n3;
    O.dis[g] = (0.5 * G.dx[t] * fabs(n1) + 0.5 * G.dy[t] * fabs(n2) + 0.5 * G.dz[t] * fabs(n3)) - d1;
}

__global__ void __launch_bounds__(NB_THREADS) k_normals(const __grid_constant__ Dims D, const __grid_constant__ Geo G,
                                                        const double *__restrict__ vfl,
                                                        const double *__restrict__ phi, NormalOut O,
                                                        const uint32_t *__restrict__ list,
                                                        const unsigned *__restrict__ count)
{
    after_previous();
    if (blockIdx.x < kNormalBlocks) {
        // 32 neighbouring entries to a warp, a warp of every block before the next
        // of any: a short list is spread over all SMs
        const unsigned n = *count;
        for (unsigned long long q = (unsigned long long)(threadIdx.x >> 5) * kNormalBlocks * 32 + blockIdx.x * 32 +
                                    (threadIdx.x & 31);
             q < n; q += (unsigned long long)kNormalBlocks * NB_THREADS) {
            int i, j, k;
            tr::cell_of(D, list[q], i, j, k);
            normal_cell(D, G, vfl, phi, O, i, j, k);
        }
        return;
    }
    const unsigned long long rows = (unsigned long long)D.J * D.K;
    for (unsigned long long r = blockIdx.x - kNormalBlocks; r < rows; r += gridDim.x - kNormalBlocks) {
        const int j = (int)(r % D.J) + 1, k = (int)(r / D.J) + 1;
        for (int i = threadIdx.x + 1; i <= D.I; i += NB_THREADS) {
            const size_t g = D.g(i, j, k), n = D.n(i, j, k);
            const double v = vfl[g];
            const bool bulk = tr::is_plus_zero(v) || tr::is_one(v);
            O.key[n] = (unsigned long long)tr::key_of(1.0e4);
            O.fix[n] = 0;
            O.cls[n] = (uint8_t)((bulk || tr::band_target(v) ? 1 : 0) | (tr::hi32(phi[g]) >> 31 ? 2 : 0));
            O.ub[n] = __float_as_uint(tr::BAND_UB);
            if (!bulk && tr::partial_cell(v)) continue;   // listed
            if (tr::is_interface(D, vfl, i, j, k)) {
                normal_cell(D, G, vfl, phi, O, i, j, k);
            } else {
                O.nxl[g] = 0.0;
                O.nyl[g] = 0.0;
                O.nzl[g] = 0.0;
            }
        }
    }
}

// One directional sweep (tr::line_face, tr::line_update), which also lists the
// cells it leaves partly filled.  Along x a thread computes its cell's high
// face and takes the low one from its neighbour through shared memory; along y
// and z it marches `len` cells of its line and carries the face between two of
// them.  Bound: the FP64 pipe (about 20 operations per bulk cell, where faces
// computed for both neighbours and quotients formed anew took 60), at 128^3
// 0.12-0.16 ms per sweep against 0.28-0.44 ms before; on small grids the
// latency of the chain along a line.
constexpr int SW_X = 256;   // most threads of an x-sweep block

template <bool LATER>
__global__ void __launch_bounds__(SW_X) k_sweep_x(const __grid_constant__ Dims D, const __grid_constant__ Geo G,
                                                  const __grid_constant__ tr::SweepIn S, const double *__restrict__ flo,
                                                  const double *__restrict__ fhi, double *__restrict__ vf_out,
                                                  double *__restrict__ ls_out, uint32_t *__restrict__ list,
                                                  unsigned *__restrict__ count)
{
    after_previous();
    __shared__ tr::LineFace sh[SW_X];
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z + 1;
    const bool in = i <= D.I && j <= D.J;
    tr::LineStep s;
    tr::LineFace hi, lo;
    if (in) {
        s = tr::line_step(G.dx[D.n(i, j, k)], S.dtv);
        hi = tr::line_face(D, G, S, 0, s, G.dx, G.x, flo, fhi, i, j, k);
        sh[tid] = hi;
    }
    __syncthreads();
    bool part = false;
    if (in) {
        if (threadIdx.x > 0) {
            lo = sh[tid - 1];
        } else if (i > 1) {
            const tr::LineStep sl = tr::line_step(G.dx[D.n(i - 1, j, k)], S.dtv);
            lo = tr::line_face(D, G, S, 0, sl, G.dx, G.x, flo, fhi, i - 1, j, k);
        } else {
            lo = tr::LineFace{0.0, 0.0, 0.0, 0.0, 0.0};
        }
        double a, b;
        tr::line_update<LATER>(D, S, 0, s, lo, hi, i, j, k, a, b);
        const size_t t = D.g(i, j, k);
        vf_out[t] = a;
        ls_out[t] = b;
        part = tr::partial_cell(a);
    }
    append(part, in ? (uint32_t)D.n(i, j, k) : 0u, list, count);
}

template <int AX, bool LATER>
__global__ void __launch_bounds__(NX) k_sweep_yz(const __grid_constant__ Dims D, const __grid_constant__ Geo G,
                                                 const __grid_constant__ tr::SweepIn S, const double *__restrict__ flo,
                                                 const double *__restrict__ fhi, double *__restrict__ vf_out,
                                                 double *__restrict__ ls_out, uint32_t *__restrict__ list,
                                                 unsigned *__restrict__ count, int len)
{
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int o = blockIdx.y * blockDim.y + threadIdx.y + 1;   // the other index: k or j
    const bool in = i <= D.I && o <= (AX == 1 ? D.K : D.J);
    const int n = D.len(AX), m0 = blockIdx.z * len + 1, m1 = min(m0 + len - 1, n);
    const double *d = AX == 1 ? G.dy : G.dz, *c = AX == 1 ? G.y : G.z;
    tr::LineStep s;
    tr::LineFace lo = tr::LineFace{0.0, 0.0, 0.0, 0.0, 0.0};
    if (in) {
        const int m = m0 >= 2 ? m0 - 1 : m0;
        s = tr::line_step(d[tr::line_n(D, AX, m, i, o)], S.dtv);
        if (m0 >= 2) lo = tr::line_face(D, G, S, AX, s, d, c, flo, fhi, m, i, o);
    }
    for (int m = m0; m <= m1; ++m) {
        bool part = false;
        const int j = AX == 1 ? m : o, k = AX == 1 ? o : m;
        if (in) {
            const double dm = d[tr::line_n(D, AX, m, i, o)];
            if (!tr::same_bits(dm, s.d)) s = tr::line_step(dm, S.dtv);
            const tr::LineFace hi = tr::line_face(D, G, S, AX, s, d, c, flo, fhi, m, i, o);
            double a, b;
            tr::line_update<LATER>(D, S, AX, s, lo, hi, m, i, o, a, b);
            const size_t t = D.g(i, j, k);
            vf_out[t] = a;
            ls_out[t] = b;
            part = tr::partial_cell(a);
            lo = hi;
        }
        append(part, in ? (uint32_t)D.n(i, j, k) : 0u, list, count);
    }
}

// BoundaryConditionLvsVof: blockIdx.y is the axis, x strides its planes.
__global__ void k_walls(Dims D, Geo G, tr::WallIn W)
{
    after_previous();
    const int axis = blockIdx.y;
    const size_t np = D.plane_size(axis);
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < np; t += (size_t)gridDim.x * blockDim.x)
        tr::wall_point(D, G, W, axis, t);
}

// The band pairs: a warp takes a third of one listed cell's 729 offsets at a
// time, 32 offsets at once.
constexpr int BP_PARTS = 3, BP_PART = tr::BAND_CELLS / BP_PARTS, BP_THREADS = 256, BP_WARPS = BP_THREADS / 32;
static_assert(BP_PARTS * BP_PART == tr::BAND_CELLS, "whole parts");

struct BandItem {
    int i, j, k;
    tr::BandSource B;
};
// A listed cell for a warp, its faces in F (shared memory of the warp); false
// if it is no interface cell.  Lane q < 7 converts one of the cell's seven
// values (one FP64 conversion per warp), the others get it by shuffle.
__device__ __forceinline__ bool band_item(const Dims &D, const Geo &G, const double *vfl, const double *nx,
                                          const double *ny, const double *nz, const double *dis, uint32_t c,
                                          tr::BandFace *F, BandItem &w)
{
    tr::cell_of(D, c, w.i, w.j, w.k);
    const size_t g = D.g(w.i, w.j, w.k);
    if (!tr::band_interface(vfl[g])) return false;
    const int lane = threadIdx.x & 31;
    const double *p = lane == 0 ? nx + g : lane == 1 ? ny + g : lane == 2 ? nz + g : lane == 3 ? dis + g
                    : lane == 4 ? G.dx + c : lane == 5 ? G.dy + c : G.dz + c;
    const float f = (float)*p;
    float v[7];
#pragma unroll
    for (int q = 0; q < 7; ++q) v[q] = __shfl_sync(0xffffffffu, f, q);
    w.B = tr::band_source(v[0], v[1], v[2], v[3], v[4], v[5], v[6]);
    __syncwarp();   // the last item's faces have been read
    if (lane < 6) F[lane] = tr::band_face(w.B, lane);
    __syncwarp();
    return true;
}
// The target of offset t, if it is one: its interior index, its class byte.
__device__ __forceinline__ bool band_target_of(const Dims &D, const BandItem &w, const uint8_t *cls, int t, int &ii,
                                               int &jj, int &kk, size_t &tc, uint8_t &cl)
{
    tr::band_offset(t, ii, jj, kk);
    const int ti = w.i + ii, tj = w.j + jj, tk = w.k + kk;
    if (!(1 <= ti && ti <= D.I && 1 <= tj && tj <= D.J && 1 <= tk && tk <= D.K)) return false;
    tc = D.n(ti, tj, tk);
    cl = cls[tc];
    return cl & 1;
}

// Pass 1: every target of a pair is marked and keeps the least FP32 upper
// bound of its distances.
__global__ void __launch_bounds__(BP_THREADS) k_band_bound(Dims D, Geo G, const double *__restrict__ vfl,
                                                           const double *__restrict__ nx, const double *__restrict__ ny,
                                                           const double *__restrict__ nz,
                                                           const double *__restrict__ dis,
                                                           const uint8_t *__restrict__ cls,
                                                           const uint32_t *__restrict__ list,
                                                           const unsigned *__restrict__ count, unsigned *ub,
                                                           uint8_t *fix)
{
    after_previous();
    __shared__ tr::BandFace faces[BP_WARPS][6];
    const unsigned long long items = (unsigned long long)*count * BP_PARTS;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const unsigned long long nw = (unsigned long long)gridDim.x * BP_WARPS;
    for (unsigned long long m = (unsigned long long)blockIdx.x * BP_WARPS + wp; m < items; m += nw) {
        BandItem w;
        if (!band_item(D, G, vfl, nx, ny, nz, dis, list[m / BP_PARTS], faces[wp], w)) continue;
        const int t0 = (int)(m % BP_PARTS) * BP_PART;
        for (int t = t0 + lane; t < t0 + BP_PART; t += 32) {
            int ii, jj, kk;
            size_t tc;
            uint8_t cl;
            if (!band_target_of(D, w, cls, t, ii, jj, kk, tc, cl)) continue;
            fix[tc] = 1;
            float lo, hi;
            if (tr::band_bounds(w.B, faces[wp], ii, jj, kk, cl & 2, lo, hi) && hi < __uint_as_float(ub[tc]))
                atomicMin(ub + tc, __float_as_uint(hi));
        }
    }
}

// Out of line: its registers would otherwise set the whole pass's, which waits
// on memory and wants warps in flight.
__device__ __noinline__ void band_pair_fp64(const Dims &D, const Geo &G, const double *vfl, const double *phi,
                                            const double *nx, const double *ny, const double *nz, const double *dis,
                                            uint32_t c, int t, unsigned long long *key, uint8_t *fix)
{
    int i, j, k;
    tr::cell_of(D, c, i, j, k);
    tr::band_pair(D, G, vfl, phi, nx, ny, nz, dis, i, j, k, t, key, fix);
}

// Pass 2: the pairs that may hold their target's minimum -- lower bound not
// above the target's least upper bound, or no bounds; about one in 65 on a
// sphere -- collect in the block's queue and are computed in FP64 a warp full
// at a time.  Its rounds are the block's: each warp takes at most one item,
// then the queue is emptied if it may not hold the next round's.
constexpr int BQ_CAP = 4096, BQ_ROUND = BP_WARPS * BP_PART;

__global__ void __launch_bounds__(BP_THREADS, 4) k_band_pairs(const __grid_constant__ Dims D, const __grid_constant__ Geo G,
                                                              const double *__restrict__ vfl,
                                                              const double *__restrict__ phi,
                                                              const double *__restrict__ nx,
                                                              const double *__restrict__ ny,
                                                              const double *__restrict__ nz,
                                                              const double *__restrict__ dis,
                                                              const uint8_t *__restrict__ cls,
                                                              const uint32_t *__restrict__ list,
                                                              const unsigned *__restrict__ count,
                                                              const unsigned *__restrict__ ub, unsigned long long *key,
                                                              uint8_t *fix)
{
    after_previous();
    __shared__ tr::BandFace faces[BP_WARPS][6];
    __shared__ uint32_t q_cell[BQ_CAP];
    __shared__ unsigned short q_off[BQ_CAP];
    __shared__ int q_count;
    const unsigned long long items = (unsigned long long)*count * BP_PARTS;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (threadIdx.x == 0) q_count = 0;
    __syncthreads();
    auto empty = [&](int n) {
        for (int q = threadIdx.x; q < n; q += BP_THREADS)
            band_pair_fp64(D, G, vfl, phi, nx, ny, nz, dis, q_cell[q], q_off[q], key, fix);
    };
    for (unsigned long long m0 = (unsigned long long)blockIdx.x * BP_WARPS; m0 < items;
         m0 += (unsigned long long)gridDim.x * BP_WARPS) {
        const unsigned long long m = m0 + wp;
        BandItem w;
        const uint32_t c = m < items ? list[m / BP_PARTS] : 0u;
        if (m < items && band_item(D, G, vfl, nx, ny, nz, dis, c, faces[wp], w)) {
            const int t0 = (int)(m % BP_PARTS) * BP_PART;
            for (int tb = t0; tb < t0 + BP_PART; tb += 32) {
                const int t = tb + lane;
                int ii, jj, kk;
                size_t tc;
                uint8_t cl;
                bool need = false;
                if (t < t0 + BP_PART && band_target_of(D, w, cls, t, ii, jj, kk, tc, cl)) {
                    float lo, hi;
                    need = !(tr::band_bounds(w.B, faces[wp], ii, jj, kk, cl & 2, lo, hi) &&
                             lo > __uint_as_float(ub[tc]));
                }
                const unsigned mask = __ballot_sync(0xffffffffu, need);
                if (!mask) continue;
                int base = 0;
                if (lane == 0) base = atomicAdd(&q_count, __popc(mask));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (need) {
                    const int at = base + __popc(mask & ((1u << lane) - 1u));
                    q_cell[at] = c;
                    q_off[at] = (unsigned short)t;
                }
            }
        }
        __syncthreads();
        const int n = q_count;
        if (n > BQ_CAP - BQ_ROUND) {
            empty(n);
            __syncthreads();
            if (threadIdx.x == 0) q_count = 0;
        }
        __syncthreads();
    }
    empty(q_count);
}

__global__ void k_band_value(Dims D, Geo G, const double *__restrict__ vfl, const double *__restrict__ dis,
                             const unsigned long long *__restrict__ key, const uint8_t *__restrict__ fix,
                             double *phi)
{
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y + 1, k = blockIdx.z + 1;
    if (i > D.I) return;
    phi[D.g(i, j, k)] = tr::band_value(D, G, vfl, dis, i, j, k, key, fix);
}

// ComputeUVWLiquidField for one family over its ghosted grid: the cells of
// (0:I-1,0:J-1,0:K-1) take the direction averages, the interior cells the
// liquid fraction.
__global__ void k_uvw(Dims D, int fam, Geo G, const double *__restrict__ phil, const double *__restrict__ nxl,
                      const double *__restrict__ nyl, const double *__restrict__ nzl, const double *__restrict__ vofl,
                      const double *__restrict__ vdx, const double *__restrict__ vdy, const double *__restrict__ vdz,
                      double *o_phil, double *o_nxl, double *o_nyl, double *o_nzl, double *o_vofl)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
    if (i > D.I + 1) return;
    const double *pin[4] = {phil, nxl, nyl, nzl};
    const double *d = fam == 0 ? G.dx : fam == 1 ? G.dy : G.dz;
    const size_t t = D.g(i, j, k);
    if (i < D.I && j < D.J && k < D.K) {
        double av[4];
        tr::family_average(D, fam, d, pin, i, j, k, av);
        o_phil[t] = av[0];
        o_nxl[t] = av[1];
        o_nyl[t] = av[2];
        o_nzl[t] = av[3];
    }
    if (i >= 1 && i <= D.I && j >= 1 && j <= D.J && k >= 1 && k <= D.K)
        o_vofl[t] = tr::family_vofl(D, fam, G.dx, G.dy, G.dz, phil, nxl, nyl, nzl, vofl, vdx, vdy, vdz, i, j, k);
}

// ---- one time step ---------------------------------------------------------

int launch_check(scf_clsvof_ctx *ctx, const char *what)
{
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        tr_err(ctx, "%s launch: %s", what, cudaGetErrorString(e));
        return SCF_ERR_CUDA;
    }
    return SCF_OK;
}

// With timing on, an event pair around each launch, tagged with its kind
// (0 reconstruct, 1 sweep, 2 walls, 3 redistancing).
struct Timer {
    scf_clsvof_ctx *ctx;
    int n = 0;
    void before(int kind)
    {
        if (!ctx->timing || (size_t)(2 * n + 1) >= ctx->tev.size()) return;
        cudaEventRecord(ctx->tev[2 * n], ctx->st);
        ctx->tkind[n] = kind;
    }
    void after()
    {
        if (!ctx->timing || (size_t)(2 * n + 1) >= ctx->tev.size()) return;
        cudaEventRecord(ctx->tev[2 * n + 1], ctx->st);
        ++n;
    }
};

// Blocks of the two band passes, whose warps loop over the listed cells.
constexpr int kBandBlocks = 152 * 4;
// Single-warp blocks of k_partial_fluxes.
constexpr int kFluxBlocks = 152 * 8;

// Threads along i of a block of at most `most` threads that takes whole warps
// of one or several lines.
int line_threads(int I, int most) { return std::min(most, (I + 31) / 32 * 32); }

// Cells a thread of the y and z sweeps marches: a face is computed once per
// thread start beyond the cells' own, so the longest of 16, 8, 4, 2 that gives
// four blocks to each SM.
int sweep_len(int n, long long line_blocks)
{
    int len = 16;
    while (len > 2 && line_blocks * ((n + len - 1) / len) < 152 * 4) len /= 2;
    return len;
}

// Clsvof_Scheme (Clsvof.f90:355-798) on the staged state; counts launches.
// listed: the step before, in the same call, left the list of partial cells
// (between calls the caller may write the fields).
int scheme_step(scf_clsvof_ctx *ctx, bool listed, int &launches, Timer &T)
{
    const Dims D = ctx->D;
    const Geo G = geo_of(ctx);
    const double dtv = ctx->dt / (double)tr::NSUB;
    const dim3 gin((D.I + NX - 1) / NX, D.J, D.K);   // interior cells
    size_t pmax = std::max(D.plane_size(0), std::max(D.plane_size(1), D.plane_size(2)));
    int rc;
    // 18 sweeps, an even number: the last one's list is where the first looks
    static_assert((3 * tr::NSUB) % 2 == 0, "list buffers alternate");
    if (listed &&
        cudaMemcpyAsync(ctx->npart, ctx->npart + 3 * tr::NSUB, sizeof(unsigned), cudaMemcpyDeviceToDevice, ctx->st) !=
            cudaSuccess)
        return launch_check(ctx, "cudaMemcpyAsync");
    if (cudaMemsetAsync(ctx->npart + 1, 0, 3 * tr::NSUB * sizeof(unsigned), ctx->st) != cudaSuccess)
        return launch_check(ctx, "cudaMemsetAsync");
    for (int kk = 1; kk <= tr::NSUB; ++kk) {
        const int first = kk % 3 == 0 ? 0 : kk % 3 == 1 ? 1 : 2;
        int cur = 0;
        for (int s = 0; s < 3; ++s) {
            const int ax = (first + s) % 3, out = s == 0 ? 1 : s == 1 ? 2 : 0;
            tr::SweepIn S{};
            S.vfl = ctx->vf[cur];
            S.phi = ctx->ls[cur];
            S.vel = ctx->vel[ax];
            S.bc_vel = ctx->bc_vel[ax];
            S.bc_lvs = ctx->lvs_bc[2 * ax];
            S.vf_first = ctx->vf[1];
            S.ls_first = ctx->ls[1];
            S.dtv = dtv;
            S.axis = ax;
            S.stage = s;
            // the list this sweep writes and the one the sweep before left
            const int sw = 3 * (kk - 1) + s;
            uint32_t *list = ctx->part[(sw + 1) & 1];
            unsigned *count = ctx->npart + sw + 1;
            T.before(0);
            if (sw == 0 && !listed)
                launch_after(k_partial_fluxes_scan, rb_grid(D), RB_THREADS, 0, ctx->st, D, G, S, ctx->flo, ctx->fhi);
            else
                launch_after(k_partial_fluxes, kFluxBlocks, 32, 0, ctx->st, D, G, S, ctx->part[sw & 1], ctx->npart + sw, ctx->flo,
                                                                  ctx->fhi);
            T.after();
            if ((rc = launch_check(ctx, "k_partial_fluxes")) != SCF_OK) return rc;
            T.before(1);
            if (ax == 0) {
                const int bx = line_threads(D.I, SW_X), by = SW_X / bx;
                launch_after(s ? k_sweep_x<true> : k_sweep_x<false>, dim3((D.I + bx - 1) / bx, (D.J + by - 1) / by, D.K), dim3(bx, by), 0, ctx->st, 
                    D, G, S, ctx->flo, ctx->fhi, ctx->vf[out], ctx->ls[out], list, count);
            } else {
                const int bx = line_threads(D.I, NX), by = NX / bx, n = D.len(ax);
                dim3 g((D.I + bx - 1) / bx, ((ax == 1 ? D.K : D.J) + by - 1) / by);
                const int len = sweep_len(n, (long long)g.x * g.y);
                g.z = (n + len - 1) / len;
                auto *kernel = ax == 1 ? (s ? k_sweep_yz<1, true> : k_sweep_yz<1, false>)
                                       : (s ? k_sweep_yz<2, true> : k_sweep_yz<2, false>);
                launch_after(kernel, g, dim3(bx, by), 0, ctx->st, D, G, S, ctx->flo, ctx->fhi, ctx->vf[out], ctx->ls[out], list, count,
                                              len);
            }
            T.after();
            if ((rc = launch_check(ctx, "k_sweep")) != SCF_OK) return rc;
            launches += 2;
            cur = out;
        }
        tr::WallIn W;
        W.phil = ctx->ls[0];
        W.vofl = ctx->vf[0];
        for (int q = 0; q < 2; ++q) {
            W.phil_more[q] = ctx->ls[q + 1];
            W.vofl_more[q] = ctx->vf[q + 1];
        }
        W.nxl = ctx->nxl;
        W.nx = ctx->fn[0];
        W.ny = ctx->fn[1];
        W.nz = ctx->fn[2];
        for (int f = 0; f < 6; ++f) {
            W.lvs_bc[f] = ctx->lvs_bc[f];
            W.vof_bc[f] = ctx->vof_bc[f];
            W.lvs_flag[f] = ctx->lvs_flag[f];
            W.vof_flag[f] = ctx->vof_flag[f];
            W.lvs_const[f] = ctx->lvs_const[f];
            W.vof_const[f] = ctx->vof_const[f];
        }
        T.before(2);
        launch_after(k_walls, dim3(blocks_for(pmax), 3), NT, 0, ctx->st, D, G, W);
        T.after();
        if ((rc = launch_check(ctx, "k_walls")) != SCF_OK) return rc;
        const uint32_t *list = ctx->part[(3 * kk) & 1];
        const unsigned *count = ctx->npart + 3 * kk;
        NormalOut O;
        O.nxl = ctx->nxl; O.nyl = ctx->nyl; O.nzl = ctx->nzl; O.dis = ctx->dis;
        O.key = ctx->key; O.fix = ctx->fix; O.cls = ctx->cls; O.ub = ctx->ub;
        const unsigned nb = kNormalBlocks + (unsigned)std::min<size_t>((size_t)D.J * D.K, 152 * 32);
        T.before(0);
        launch_after(k_normals, nb, NB_THREADS, 0, ctx->st, D, G, ctx->vf[0], ctx->ls[0], O, list, count);
        T.after();
        if ((rc = launch_check(ctx, "k_normals")) != SCF_OK) return rc;
        T.before(3);
        launch_after(k_band_bound, kBandBlocks, BP_THREADS, 0, ctx->st, D, G, ctx->vf[0], ctx->nxl, ctx->nyl, ctx->nzl, ctx->dis,
                                                              ctx->cls, list, count, ctx->ub, ctx->fix);
        T.after();
        if ((rc = launch_check(ctx, "k_band_bound")) != SCF_OK) return rc;
        T.before(3);
        launch_after(k_band_pairs, kBandBlocks, BP_THREADS, 0, ctx->st, D, G, ctx->vf[0], ctx->ls[0], ctx->nxl, ctx->nyl,
                                                              ctx->nzl, ctx->dis, ctx->cls, list, count, ctx->ub,
                                                              ctx->key, ctx->fix);
        T.after();
        if ((rc = launch_check(ctx, "k_band_pairs")) != SCF_OK) return rc;
        T.before(3);
        launch_after(k_band_value, gin, NX, 0, ctx->st, D, G, ctx->vf[0], ctx->dis, ctx->key, ctx->fix, ctx->ls[0]);
        T.after();
        if ((rc = launch_check(ctx, "k_band_value")) != SCF_OK) return rc;
        launches += 5;
    }
    return SCF_OK;
}

// Zeroed on the context's stream: the legacy stream does not order before it,
// and may have the caller's work queued.
template <typename P>
int alloc(scf_clsvof_ctx *ctx, P **ptr, size_t count)
{
    void *p = nullptr;
    const size_t bytes = std::max<size_t>(count * sizeof(P), 16);
    const cudaError_t e = scf_mem::dev_malloc(&p, bytes);
    if (e != cudaSuccess) {
        tr_err(ctx, "cudaMalloc(%zu bytes): %s", bytes, cudaGetErrorString(e));
        return SCF_ERR_OUT_OF_MEMORY;
    }
    ctx->mem.push_back(p);
    *ptr = (P *)p;
    return cudaMemsetAsync(p, 0, bytes, ctx->st) == cudaSuccess ? SCF_OK : SCF_ERR_CUDA;
}

float elapsed(cudaEvent_t a, cudaEvent_t b)
{
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
}

}  // namespace

extern "C" int scf_clsvof_create(scf_clsvof_ctx **out, int32_t imax, int32_t jmax, int32_t kmax, int32_t device)
{
    if (!out) return SCF_ERR_BAD_ARG;
    *out = nullptr;
    if (imax < 3 || jmax < 3 || kmax < 3 || imax > 65533 || jmax > 65533 || kmax > 65533) return SCF_ERR_BAD_ARG;
    // the redistancing lists interface cells by 32-bit interior index
    if ((unsigned long long)imax * (unsigned long long)jmax * (unsigned long long)kmax >= (1ull << 32))
        return SCF_ERR_BAD_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return SCF_ERR_NO_DEVICE;
    scf_clsvof_ctx *ctx = new scf_clsvof_ctx();
    ctx->device = device;
    ctx->D = Dims{imax, jmax, kmax};
    auto fail = [&](int rc) {
        scf_clsvof_destroy(ctx);
        return rc;
    };
    if (cudaStreamCreateWithFlags(&ctx->st, cudaStreamNonBlocking) != cudaSuccess) return fail(SCF_ERR_CUDA);
    for (auto &e : ctx->ev)
        if (cudaEventCreate(&e) != cudaSuccess) return fail(SCF_ERR_CUDA);
    const size_t nin = ctx->D.interior(), ng = ctx->D.ghosted();
    int rc;
#define TRY(ptr, count)                                         \
    if ((rc = alloc(ctx, &(ptr), (count))) != SCF_OK) return fail(rc);
    for (auto &p : ctx->geo) TRY(p, nin)
    for (int b = 0; b < 3; ++b) { TRY(ctx->vf[b], ng) TRY(ctx->ls[b], ng) }
    TRY(ctx->flo, ng) TRY(ctx->fhi, ng) TRY(ctx->dis, ng)
    TRY(ctx->nxl, ng) TRY(ctx->nyl, ng) TRY(ctx->nzl, ng)
    for (auto &p : ctx->fn) TRY(p, ng)
    for (auto &p : ctx->vel) TRY(p, ng)
    for (int a = 0; a < 3; ++a) TRY(ctx->bc_vel[a], ctx->D.plane_size(a))
    for (int f = 0; f < 6; ++f) { TRY(ctx->lvs_bc[f], ctx->D.plane_size(f / 2)) TRY(ctx->vof_bc[f], ctx->D.plane_size(f / 2)) }
    TRY(ctx->key, nin) TRY(ctx->fix, nin) TRY(ctx->cls, nin) TRY(ctx->ub, nin)
    TRY(ctx->part[0], nin) TRY(ctx->part[1], nin) TRY(ctx->npart, 3 * tr::NSUB + 1)
#undef TRY
    *out = ctx;
    return SCF_OK;
}

extern "C" int scf_clsvof_set_timing(scf_clsvof_ctx *ctx, int32_t on)
{
    if (!ctx) return SCF_ERR_BAD_ARG;
    cudaSetDevice(ctx->device);
    const size_t need = 2 * (size_t)tr::NSUB * 11;   // two events per launch of a step
    while (on && ctx->tev.size() < need) {
        cudaEvent_t e = nullptr;
        TK(cudaEventCreate(&e));
        ctx->tev.push_back(e);
    }
    ctx->tkind.assign(need / 2, 0);
    ctx->timing = on != 0;
    return SCF_OK;
}

extern "C" int scf_clsvof_destroy(scf_clsvof_ctx *ctx)
{
    if (!ctx) return SCF_ERR_BAD_ARG;
    cudaSetDevice(ctx->device);
    if (ctx->st) cudaStreamSynchronize(ctx->st);
    for (cudaEvent_t e : ctx->tev) cudaEventDestroy(e);
    for (void *p : ctx->mem) scf_mem::dev_free(p);
    for (auto &e : ctx->ev)
        if (e) cudaEventDestroy(e);
    if (ctx->st) cudaStreamDestroy(ctx->st);
    delete ctx;
    return SCF_OK;
}

extern "C" int scf_clsvof_stage(scf_clsvof_ctx *ctx, const scf_clsvof_in *in, const scf_clsvof_state *s)
{
    if (!ctx || !in || !s) return SCF_ERR_BAD_ARG;
    const double *need[] = {in->x, in->y, in->z, in->dx, in->dy, in->dz, in->u, in->v, in->w, in->nx, in->ny,
                            in->nz, in->bc_u_w, in->bc_v_s, in->bc_w_b, s->vofl, s->phil, s->nxl, s->nyl, s->nzl};
    for (const double *p : need)
        if (!p) {
            tr_err(ctx, "scf_clsvof_stage: a required array is null");
            return SCF_ERR_BAD_ARG;
        }
    for (int f = 0; f < 6; ++f)
        if (!s->lvs_bc[f]) {
            tr_err(ctx, "scf_clsvof_stage: lvs_bc[%d] is null", f);
            return SCF_ERR_BAD_ARG;
        }
    if (!(in->dt >= 0.0) || !std::isfinite(in->dt)) {
        tr_err(ctx, "scf_clsvof_stage: dt must be finite and >= 0");
        return SCF_ERR_BAD_ARG;
    }
    cudaSetDevice(ctx->device);
    const size_t nin = ctx->D.interior(), ng = ctx->D.ghosted();
    const size_t bi = nin * sizeof(double), bg = ng * sizeof(double);
    const double *geo[6] = {in->x, in->y, in->z, in->dx, in->dy, in->dz};
    for (int q = 0; q < 6; ++q) TK(stage_h2d(ctx->geo[q], geo[q], bi, ctx->st, 0, nullptr, nullptr));
    const double *vel[3] = {in->u, in->v, in->w}, *fn[3] = {in->nx, in->ny, in->nz};
    const double *bcv[3] = {in->bc_u_w, in->bc_v_s, in->bc_w_b};
    for (int a = 0; a < 3; ++a) {
        TK(stage_h2d(ctx->vel[a], vel[a], bg, ctx->st, 0, nullptr, nullptr));
        TK(stage_h2d(ctx->fn[a], fn[a], bg, ctx->st, 0, nullptr, nullptr));
        TK(stage_h2d(ctx->bc_vel[a], bcv[a], ctx->D.plane_size(a) * sizeof(double), ctx->st, 0, nullptr, nullptr));
    }
    TK(stage_h2d(ctx->vf[0], s->vofl, bg, ctx->st, 0, nullptr, nullptr));
    TK(stage_h2d(ctx->ls[0], s->phil, bg, ctx->st, 0, nullptr, nullptr));
    for (int b = 1; b < 3; ++b) {   // the ping-pong buffers' ghosts must match buffer 0's
        TK(cudaMemcpyAsync(ctx->vf[b], ctx->vf[0], bg, cudaMemcpyDeviceToDevice, ctx->st));
        TK(cudaMemcpyAsync(ctx->ls[b], ctx->ls[0], bg, cudaMemcpyDeviceToDevice, ctx->st));
    }
    TK(stage_h2d(ctx->nxl, s->nxl, bg, ctx->st, 0, nullptr, nullptr));
    TK(stage_h2d(ctx->nyl, s->nyl, bg, ctx->st, 0, nullptr, nullptr));
    TK(stage_h2d(ctx->nzl, s->nzl, bg, ctx->st, 0, nullptr, nullptr));
    for (int f = 0; f < 6; ++f)
        TK(cudaMemcpyAsync(ctx->lvs_bc[f], s->lvs_bc[f], ctx->D.plane_size(f / 2) * sizeof(double),
                           cudaMemcpyHostToDevice, ctx->st));
    for (int f = 0; f < 6; ++f) {
        ctx->lvs_flag[f] = in->lvs_flag[f];
        ctx->vof_flag[f] = in->vof_flag[f];
        ctx->lvs_const[f] = in->lvs_const[f];
        ctx->vof_const[f] = in->vof_const[f];
    }
    ctx->dt = in->dt;
    TK(cudaStreamSynchronize(ctx->st));
    ctx->staged = true;
    return SCF_OK;
}

extern "C" int scf_clsvof_run(scf_clsvof_ctx *ctx, int32_t steps, scf_clsvof_stats *stats)
{
    if (!ctx || steps < 0) return SCF_ERR_BAD_ARG;
    if (!ctx->staged) {
        tr_err(ctx, "scf_clsvof_run: nothing staged");
        return SCF_ERR_BAD_ARG;
    }
    cudaSetDevice(ctx->device);
    int launches = 0, rc;
    double ms_kind[4] = {0.0, 0.0, 0.0, 0.0};
    TK(cudaEventRecord(ctx->ev[0], ctx->st));
    for (int n = 0; n < steps; ++n) {
        Timer T{ctx};
        if ((rc = scheme_step(ctx, n > 0, launches, T)) != SCF_OK) return rc;
        if (ctx->timing) {
            TK(cudaStreamSynchronize(ctx->st));
            for (int q = 0; q < T.n; ++q) ms_kind[ctx->tkind[q]] += elapsed(ctx->tev[2 * q], ctx->tev[2 * q + 1]);
        }
    }
    TK(cudaEventRecord(ctx->ev[1], ctx->st));
    TK(cudaStreamSynchronize(ctx->st));
    if (stats) {
        stats->ms_run = elapsed(ctx->ev[0], ctx->ev[1]);
        stats->steps = steps;
        stats->gpu_launches = launches;
        for (int q = 0; q < 4; ++q) stats->ms_kernels[q] = ms_kind[q];
    }
    return SCF_OK;
}

extern "C" int scf_clsvof_fetch(scf_clsvof_ctx *ctx, scf_clsvof_state *s, scf_clsvof_stats *stats)
{
    if (!ctx || !s) return SCF_ERR_BAD_ARG;
    if (!ctx->staged) {
        tr_err(ctx, "scf_clsvof_fetch: nothing staged");
        return SCF_ERR_BAD_ARG;
    }
    double *need[] = {s->vofl, s->phil, s->nxl, s->nyl, s->nzl};
    for (double *p : need)
        if (!p) return SCF_ERR_BAD_ARG;
    for (int f = 0; f < 6; ++f)
        if (!s->lvs_bc[f] || !s->vof_bc[f]) return SCF_ERR_BAD_ARG;
    cudaSetDevice(ctx->device);
    const size_t bg = ctx->D.ghosted() * sizeof(double);
    TK(cudaEventRecord(ctx->ev[2], ctx->st));
    TK(stage_d2h(s->vofl, ctx->vf[0], bg, ctx->st, 0, nullptr, nullptr));
    TK(stage_d2h(s->phil, ctx->ls[0], bg, ctx->st, 0, nullptr, nullptr));
    TK(stage_d2h(s->nxl, ctx->nxl, bg, ctx->st, 0, nullptr, nullptr));
    TK(stage_d2h(s->nyl, ctx->nyl, bg, ctx->st, 0, nullptr, nullptr));
    TK(stage_d2h(s->nzl, ctx->nzl, bg, ctx->st, 0, nullptr, nullptr));
    int64_t planes = 0;
    for (int f = 0; f < 6; ++f) {
        const size_t pb = ctx->D.plane_size(f / 2) * sizeof(double);
        TK(stage_d2h(s->lvs_bc[f], ctx->lvs_bc[f], pb, ctx->st, 0, nullptr, nullptr));
        TK(stage_d2h(s->vof_bc[f], ctx->vof_bc[f], pb, ctx->st, 0, nullptr, nullptr));
        planes += 2 * (int64_t)pb;
    }
    TK(cudaEventRecord(ctx->ev[3], ctx->st));
    TK(cudaStreamSynchronize(ctx->st));
    if (stats) {
        stats->ms_d2h = elapsed(ctx->ev[2], ctx->ev[3]);
        stats->bytes_d2h = 5 * (int64_t)bg + planes;
    }
    return SCF_OK;
}

extern "C" int scf_clsvof_step(scf_clsvof_ctx *ctx, const scf_clsvof_in *in, scf_clsvof_state *s,
                               scf_clsvof_stats *stats)
{
    if (!ctx) return SCF_ERR_BAD_ARG;
    scf_clsvof_stats local{};
    scf_clsvof_stats *st = stats ? stats : &local;
    *st = scf_clsvof_stats{};
    cudaSetDevice(ctx->device);
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    TK(cudaEventCreate(&t0));
    TK(cudaEventCreate(&t1));
    int rc = SCF_OK;
    cudaEventRecord(t0, ctx->st);
    if ((rc = scf_clsvof_stage(ctx, in, s)) == SCF_OK) {
        cudaEventRecord(t1, ctx->st);
        cudaEventSynchronize(t1);
        st->ms_h2d = elapsed(t0, t1);
        const size_t nin = ctx->D.interior(), ng = ctx->D.ghosted();
        int64_t planes = 0;
        for (int a = 0; a < 3; ++a) planes += (int64_t)ctx->D.plane_size(a) * 3;   // bc_vel + two lvs planes
        st->bytes_h2d = (int64_t)(6 * nin + 11 * ng) * 8 + planes * 8;
        if ((rc = scf_clsvof_run(ctx, 1, st)) == SCF_OK) rc = scf_clsvof_fetch(ctx, s, st);
    }
    cudaEventRecord(t1, ctx->st);
    cudaEventSynchronize(t1);
    st->ms_total = elapsed(t0, t1);
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    return rc;
}

extern "C" int scf_clsvof_uvw_liquid_field(scf_clsvof_ctx *ctx, const scf_clsvof_vcell cells[3],
                                           scf_clsvof_stats *stats)
{
    if (!ctx || !cells) return SCF_ERR_BAD_ARG;
    if (!ctx->staged) {
        tr_err(ctx, "scf_clsvof_uvw_liquid_field: nothing staged");
        return SCF_ERR_BAD_ARG;
    }
    for (int f = 0; f < 3; ++f) {
        const scf_clsvof_vcell &c = cells[f];
        if (!c.dx || !c.dy || !c.dz || !c.phil || !c.nxl || !c.nyl || !c.nzl || !c.vofl) {
            tr_err(ctx, "scf_clsvof_uvw_liquid_field: a required array of family %d is null", f);
            return SCF_ERR_BAD_ARG;
        }
    }
    cudaSetDevice(ctx->device);
    const size_t nin = ctx->D.interior(), ng = ctx->D.ghosted();
    int rc;
    for (int f = 0; f < 3; ++f) {
        for (auto &p : ctx->vgeo[f])
            if (!p && (rc = alloc(ctx, &p, nin)) != SCF_OK) return rc;
        for (auto &p : ctx->vfld[f])
            if (!p && (rc = alloc(ctx, &p, ng)) != SCF_OK) return rc;
    }
    TK(cudaEventRecord(ctx->ev[0], ctx->st));
    for (int f = 0; f < 3; ++f) {
        const scf_clsvof_vcell &c = cells[f];
        const double *g[3] = {c.dx, c.dy, c.dz};
        double *h[5] = {c.phil, c.nxl, c.nyl, c.nzl, c.vofl};
        for (int q = 0; q < 3; ++q)
            TK(stage_h2d(ctx->vgeo[f][q], g[q], nin * sizeof(double), ctx->st, 0, nullptr, nullptr));
        for (int q = 0; q < 5; ++q)
            TK(stage_h2d(ctx->vfld[f][q], h[q], ng * sizeof(double), ctx->st, 0, nullptr, nullptr));
    }
    TK(cudaEventRecord(ctx->ev[1], ctx->st));
    const Geo G = geo_of(ctx);
    for (int f = 0; f < 3; ++f) {
        const dim3 gg((ctx->D.I + 2 + NX - 1) / NX, ctx->D.J + 2, ctx->D.K + 2);   // ghosted cells
        k_uvw<<<gg, NX, 0, ctx->st>>>(ctx->D, f, G, ctx->ls[0], ctx->nxl, ctx->nyl, ctx->nzl, ctx->vf[0],
                                                 ctx->vgeo[f][0], ctx->vgeo[f][1], ctx->vgeo[f][2], ctx->vfld[f][0],
                                                 ctx->vfld[f][1], ctx->vfld[f][2], ctx->vfld[f][3], ctx->vfld[f][4]);
        if ((rc = launch_check(ctx, "k_uvw")) != SCF_OK) return rc;
    }
    TK(cudaEventRecord(ctx->ev[2], ctx->st));
    for (int f = 0; f < 3; ++f) {
        const scf_clsvof_vcell &c = cells[f];
        double *h[5] = {c.phil, c.nxl, c.nyl, c.nzl, c.vofl};
        for (int q = 0; q < 5; ++q)
            TK(stage_d2h(h[q], ctx->vfld[f][q], ng * sizeof(double), ctx->st, 0, nullptr, nullptr));
    }
    TK(cudaEventRecord(ctx->ev[3], ctx->st));
    TK(cudaStreamSynchronize(ctx->st));
    if (stats) {
        *stats = scf_clsvof_stats{};
        stats->ms_h2d = elapsed(ctx->ev[0], ctx->ev[1]);
        stats->ms_run = elapsed(ctx->ev[1], ctx->ev[2]);
        stats->ms_d2h = elapsed(ctx->ev[2], ctx->ev[3]);
        stats->ms_total = elapsed(ctx->ev[0], ctx->ev[3]);
        stats->bytes_h2d = (int64_t)(3 * (3 * nin + 5 * ng)) * 8;
        stats->bytes_d2h = (int64_t)(15 * ng) * 8;
        stats->gpu_launches = 3;
    }
    return SCF_OK;
}

extern "C" int scf_clsvof_device_fields(scf_clsvof_ctx *ctx, double **vofl, double **phil)
{
    if (!ctx || !vofl || !phil) return SCF_ERR_BAD_ARG;
    *vofl = ctx->staged ? ctx->vf[0] : nullptr;
    *phil = ctx->staged ? ctx->ls[0] : nullptr;
    return SCF_OK;
}

extern "C" int scf_clsvof_last_error(scf_clsvof_ctx *ctx, char *buf, size_t n)
{
    if (!ctx || !buf || n == 0) return SCF_ERR_BAD_ARG;
    snprintf(buf, n, "%s", ctx->err);
    return SCF_OK;
}
