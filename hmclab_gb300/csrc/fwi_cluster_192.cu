// Elastic shots on chip for grids of 129 to 192 columns.
#include "fwi_cluster_adjoint.cuh"
#include "fwi_cluster_forward.cuh"

namespace hmc {
namespace fwi {
template int cluster_forward_at<192>(const ShotForward&, const Waves&, bool, Strip*, cudaStream_t);
template int cluster_adjoint_at<192>(const ShotAdjoint&, bool, Strip*, cudaStream_t);
}  // namespace fwi
}  // namespace hmc
