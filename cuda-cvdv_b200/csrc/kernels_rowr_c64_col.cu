// k_rowr on columns of complex64 states (one translation unit each, so they build in parallel).
#include "rowr.cuh"

namespace cvdv {
template cudaError_t launch_rowr<float2, true>(Context*, const void*, void*, const RowProgram&, int);
}  // namespace cvdv
