// ft_hexgp_f64.cu -- double instantiations of the eight-lane C3D8 pass and their launchers.
#include "ft_hexgp.cuh"
#include "ft_launch.h"

namespace ftgpu {

int launch_hexgp(int mat, int gp, int nblocks, int threads, size_t smem, cudaStream_t s,
                 const ElemArgs<double> &A, int pass) {
  if (nblocks <= 0) return 0;
  return hexgp_by_mat<double>(mat, gp, nblocks, threads, smem, s, A, pass);
}

int launch_hexgp_geo(int nblocks, cudaStream_t s, const ElemArgs<double> &A, double *geo) {
  if (nblocks <= 0) return 0;
  k_hexgp_geo<double><<<nblocks, kHexGpThreads, 0, s>>>(A, geo);
  return (int)cudaGetLastError();
}

}  // namespace ftgpu
