// Residual suite kernels, N_b <= 16.
#include "residual_rows.cuh"

namespace qcl {

template <typename RS> int launch_residual_rows_small(const ResidualArgs<RS>& a, cudaStream_t st) {
  return padded_size(a.N) == 8 ? launch_residual_rows_t<RS, 8, 8>(a, st) : launch_residual_rows_t<RS, 16, 2>(a, st);
}
template int launch_residual_rows_small<double>(const ResidualArgs<double>&, cudaStream_t);
template int launch_residual_rows_small<float>(const ResidualArgs<float>&, cudaStream_t);

}  // namespace qcl
