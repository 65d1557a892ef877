// FP64 instantiation of the point kernels.
#include "point_kernels.cuh"

namespace pnamp {
template cudaError_t launch_points_z<zc, false>(const Params &, int, const double *, zc *, int, double *, int *,
                                                cudaStream_t, const int2 *, long long, double *, double *, double *, int);
template cudaError_t launch_multi_z<zc>(const MultiArgs &, const int4 *, int, int, int *, zc *, int, int, cudaStream_t);
template const void *point_fn<zc, false>();
template const void *multi_fn<zc>();
}  // namespace pnamp
