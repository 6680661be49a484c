// plane kernel, FP64 instantiation (see plane.cuh)
#include "plane.cuh"
namespace opfc {
template int launch_plane<double>(int, const PlaneArgs &, cudaStream_t);
template int launch_plane_fft<double>(int, const PlaneArgs &, cudaStream_t);
template int launch_z_ref<double>(int, const ZRefArgs &, cudaStream_t);
template int launch_z_adj<double>(const ZAdjArgs &, cudaStream_t);
}
