// band_arithmetic.cpp -- the checks of band_bounds.cpp, with access to the FP32
// operations the bounds are formed with on the host.
#include "band_bounds.cpp"

extern "C" float host_fma(float a, float b, float c) { return tr::band_fma(a, b, c); }
extern "C" float host_sqrt(float a) { return tr::band_sqrt(a); }
