// Fast flavour of the step kernel: the same source built with multiply-add
// contraction and approximate division (denormals kept), and the absorbing
// formulas' divisions by grid constants taken as products with reciprocals.
// The exact adjoint is built here alone: it transposes the contracted Born
// operator that the LSRTM solver applies and has no reference rounding to
// reproduce.
#define SEIS_NS fast
#define SEIS_FAST_MATH 1
#define SEIS_ADJOINT_TABLES 1
#include "fd_step_impl.cuh"

namespace seis {
namespace fast {

cudaError_t launch_adj_tables(const ShotDev *d_shots, int nshots, int max_cells, int max_tab,
                              cudaStream_t s) {
  if (nshots <= 0 || max_cells <= 0) return cudaSuccess;
  edge_coef_kernel<<<dim3((max_cells + 255) / 256, nshots), 256, 0, s>>>(d_shots, nshots);
  adj_tab_kernel<<<dim3((max_tab + 127) / 128, nshots), 128, 0, s>>>(d_shots);
  return cudaGetLastError();
}

}  // namespace fast
}  // namespace seis
