// Double-float instantiation of the point kernel that writes H/N of every gauge point.
#include "point_kernels.cuh"

namespace pnamp {
template cudaError_t launch_points_z<zd, true>(const Params &, int, const double *, zc *, int, double *, int *,
                                                cudaStream_t, const int2 *, long long, double *, double *, double *, int);
template const void *point_fn<zd, true>();
}  // namespace pnamp
