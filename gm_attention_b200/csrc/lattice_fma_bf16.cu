// bfloat16-storage instantiations of the fp32-arithmetic lattice attention kernels.
#include "lattice_fma.cuh"

namespace gmb {
namespace lat {
int lattice_pass_bf16(int mode, LatArgs& a, int n_order_rows, int64_t batch, cudaStream_t stream) {
  return lattice_pass<__nv_bfloat16>(mode, a, n_order_rows, batch, stream);
}
}  // namespace lat
}  // namespace gmb
