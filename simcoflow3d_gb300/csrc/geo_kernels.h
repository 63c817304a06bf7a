// geo_kernels.h -- device view of one cut-cell family and the launchers of
// the geometry preprocessing (k_geometry.cu).
#pragma once
#include <algorithm>
#include "scf_common.cuh"

// One cell family on the device, in the host arrays' layouts (scf_geometry.h):
// ghosted arrays of d.ng cells, interior arrays of d.n cells, ",3" arrays
// with the component as the slowest index.
struct GeoFam {
    const double *dx, *dy, *dz;           // interior
    const double *phi, *nx, *ny, *nz;     // ghosted
    double *vof, *vofl;                   // ghosted
    int *ct;                              // interior
    double *ee, *ne, *te;                 // ghosted
    double *fce, *fcn, *fct;              // ghosted x 3
    double *cent;                         // interior x 3
    double *wllh, *delh;                  // interior
    int *moex;                            // interior; nullptr: not allocated
    int *posnu;                           // (I-iu, J-iv, K-iw)
    int iu, iv, iw;
};

// Grid-stride loop over the interior cells (i, j, k 1-based).
#define INTERIOR_LOOP(d)                                                                     \
    for (int q_ = blockIdx.x * blockDim.x + threadIdx.x, i = 0, j = 0, k = 0;                 \
         q_ < (d).n && ((i = q_ % (d).I + 1), (j = (q_ / (d).I) % (d).J + 1),                 \
                        (k = q_ / ((d).I * (d).J) + 1), true);                               \
         q_ += gridDim.x * blockDim.x)

// Cells per column segment of the face kernel: the longest of 32, 16, .., 2 that
// gives two waves of its three blocks per SM.  A segment start evaluates one
// face more, a long segment is a serial chain of loads and queue barriers:
// 96^3 (host call) 10.8 ms at 32 cells, 9.7 at 4, 9.8 at 2.  Segments of two
// are not for flat grids whose columns alone give two blocks to each SM: two
// segments of four hide as much as four of two, which start twice as often
// (the four families' face kernels at 200x200x8: 0.93 ms at 8 cells, 0.89 at 4,
// 1.05 at 2; 220x220x8 0.90, 0.90 and 1.08; with K <= 6 two cells stay better,
// 300x150x6 1.00 ms at 4 cells and 0.92 at 2).
inline int geo_kseg(int I, int J, int K)
{
    const long long cols = (long long)((I + 31) / 32) * ((J + 3) / 4);
    int kseg = 32;
    while (kseg > 2 && cols * ((K + kseg - 1) / kseg) < 152 * 6) {
        if (kseg == 4 && cols >= 152 * 2 && K > 6) break;
        kseg /= 2;
    }
    return kseg;
}

// DefineCell + CellGeoCal of one family; when ev is given, ev[0] and ev[1]
// are recorded around the face kernel.
void launch_cell_geo(const GeoFam &t, const Dims &d, int *exact_count, cudaStream_t st, int *launches,
                     cudaEvent_t *ev = nullptr);
// The rest of GridPreprocess and DefineMomentumExchangeCell.
void launch_grid_preprocess_tail(const GeoFam &P, const GeoFam &U, const GeoFam &V, const GeoFam &W, const Dims &d,
                                 int *exact_count, cudaStream_t st, int *launches);
// NumberExternalCell of one family; colbuf holds (I-iu)*(J-iv) ints.
void launch_posnu(const GeoFam &t, const Dims &d, int *colbuf, int *total, cudaStream_t st, int *launches);
