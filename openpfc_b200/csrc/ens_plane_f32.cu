// ensemble plane kernel, FP32 instantiation (see ens_plane.cuh)
#include "ens_plane.cuh"
namespace opfc {
template int ens_launch_plane<float>(int, size_t, const EnsArgs &, cudaStream_t);
}
