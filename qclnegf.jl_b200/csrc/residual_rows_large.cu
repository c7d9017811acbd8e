// Residual suite kernels, N_b <= 32 (above 16).
#include "residual_rows.cuh"

namespace qcl {

template <typename RS> int launch_residual_rows_large(const ResidualArgs<RS>& a, cudaStream_t st) {
  return padded_size(a.N) == 24 ? launch_residual_rows_t<RS, 24, 2>(a, st) : launch_residual_rows_t<RS, 32, 1>(a, st);
}
template int launch_residual_rows_large<double>(const ResidualArgs<double>&, cudaStream_t);
template int launch_residual_rows_large<float>(const ResidualArgs<float>&, cudaStream_t);

}  // namespace qcl
