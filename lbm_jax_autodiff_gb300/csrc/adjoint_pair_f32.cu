#include "adjoint_pair.cuh"

namespace lbm {
template cudaError_t launch_adjoint_pair<float>(const AdjArgs<float>&, bool, cudaStream_t);
}  // namespace lbm
