// Double-float instantiation of the point kernels.
#include "point_kernels.cuh"

namespace pnamp {
template cudaError_t launch_points_z<zd, false>(const Params &, int, const double *, zc *, int, double *, int *,
                                                cudaStream_t, const int2 *, long long, double *, double *, double *, int);
template cudaError_t launch_multi_z<zd>(const MultiArgs &, const int4 *, int, int, int *, zc *, int, int, cudaStream_t);
template const void *point_fn<zd, false>();
template const void *multi_fn<zd>();
}  // namespace pnamp
