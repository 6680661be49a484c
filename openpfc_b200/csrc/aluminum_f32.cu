// Aluminum x pass, FP32 instantiation (see aluminum.cuh)
#include "aluminum.cuh"
namespace opfc {
template int launch_al_x<float>(const XLaunch &, const double *, cudaStream_t);
}
