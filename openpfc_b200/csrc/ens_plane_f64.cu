// ensemble plane kernel, FP64 instantiation (see ens_plane.cuh)
#include "ens_plane.cuh"
namespace opfc {
template int ens_launch_plane<double>(int, size_t, const EnsArgs &, cudaStream_t);
}
