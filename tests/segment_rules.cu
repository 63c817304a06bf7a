// The launch rule of the geometry's face kernel, as a library of its own.
#include "geo_kernels.h"

extern "C" int geometry_segment(int I, int J, int K) { return geo_kseg(I, J, K); }
