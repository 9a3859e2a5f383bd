// Elastic shots on chip for grids of 1 to 128 columns.
#include "fwi_cluster_adjoint.cuh"
#include "fwi_cluster_forward.cuh"

namespace hmc {
namespace fwi {
template int cluster_forward_at<128>(const ShotForward&, const Waves&, bool, Strip*, cudaStream_t);
template int cluster_adjoint_at<128>(const ShotAdjoint&, bool, Strip*, cudaStream_t);
}  // namespace fwi
}  // namespace hmc
