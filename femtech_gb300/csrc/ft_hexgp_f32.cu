// ft_hexgp_f32.cu -- float instantiations of the eight-lane C3D8 pass and their launchers.
#include "ft_hexgp.cuh"
#include "ft_launch.h"

namespace ftgpu {

int launch_hexgp(int mat, int gp, int nblocks, int threads, size_t smem, cudaStream_t s,
                 const ElemArgs<float> &A, int pass) {
  if (nblocks <= 0) return 0;
  return hexgp_by_mat<float>(mat, gp, nblocks, threads, smem, s, A, pass);
}

int launch_hexgp_geo(int nblocks, cudaStream_t s, const ElemArgs<float> &A, float *geo) {
  if (nblocks <= 0) return 0;
  k_hexgp_geo<float><<<nblocks, kHexGpThreads, 0, s>>>(A, geo);
  return (int)cudaGetLastError();
}

}  // namespace ftgpu
