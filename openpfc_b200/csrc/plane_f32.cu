// plane kernel, FP32 instantiation (see plane.cuh)
#include "plane.cuh"
namespace opfc {
template int launch_plane<float>(int, const PlaneArgs &, cudaStream_t);
template int launch_plane_fft<float>(int, const PlaneArgs &, cudaStream_t);
template int launch_z_ref<float>(int, const ZRefArgs &, cudaStream_t);
template int launch_z_adj<float>(const ZAdjArgs &, cudaStream_t);
}
