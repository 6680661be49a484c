// Aluminum x pass, FP64 instantiation (see aluminum.cuh)
#include "aluminum.cuh"
namespace opfc {
template int launch_al_x<double>(const XLaunch &, const double *, cudaStream_t);
}
