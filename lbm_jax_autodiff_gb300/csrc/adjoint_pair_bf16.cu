#include "adjoint_pair.cuh"

namespace lbm {
template cudaError_t launch_adjoint_pair<__nv_bfloat16>(const AdjArgs<float>&, bool, cudaStream_t);
}  // namespace lbm
