// k_rowr on rows of complex128 states (one translation unit each, so they build in parallel).
#include "rowr.cuh"

namespace cvdv {
template cudaError_t launch_rowr<double2, false>(Context*, const void*, void*, const RowProgram&, int);
}  // namespace cvdv
