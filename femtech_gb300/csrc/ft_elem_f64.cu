// ft_elem_f64.cu -- double instantiations of the C3D4 element kernels and the
// strain kernels, and their launchers (FP64 C3D8 elements: ft_hexgp_f64.cu).
#include "ft_elem.cuh"
#include "ft_launch.h"

namespace ftgpu {

template <int MAT>
static int go(int gp, int nb, int th, size_t sm, cudaStream_t s, const ElemArgs<double> &A, int dto) {
  if (gp == kLaunchGaussPoints)
    return launch_pdl(A.pdl, k_elem<double, 1, MAT, true, false>, nb, th, sm, s, A, dto);
  if (gp == kLaunchInjury)
    return launch_pdl(A.pdl, k_elem<double, 1, MAT, false, true>, nb, th, sm, s, A, dto);
  return launch_pdl(A.pdl, k_elem<double, 1, MAT, false, false>, nb, th, sm, s, A, dto);
}

int launch_strain_f64(int etype, int nblocks, int threads, size_t smem, cudaStream_t s,
                      const ElemArgs<double> &A, double *Eout) {
  if (nblocks <= 0) return 0;
  if (etype == 0)
    k_elem_strain<double, 0><<<nblocks, threads, smem, s>>>(A, Eout);
  else
    k_elem_strain<double, 1><<<nblocks, threads, smem, s>>>(A, Eout);
  return (int)cudaGetLastError();
}

int launch_elem_f64(int etype, int mat, int gp, int nblocks, int threads, size_t smem,
                    cudaStream_t s, const ElemArgs<double> &A, int dt_only) {
  if (nblocks <= 0) return 0;
  if (etype == 0) return (int)cudaErrorInvalidValue;
  switch (mat) {
    case 0: return go<0>(gp, nblocks, threads, smem, s, A, dt_only);
    case 1: return go<1>(gp, nblocks, threads, smem, s, A, dt_only);
    case 2: return go<2>(gp, nblocks, threads, smem, s, A, dt_only);
    case 3: return go<3>(gp, nblocks, threads, smem, s, A, dt_only);
    case 4: return go<4>(gp, nblocks, threads, smem, s, A, dt_only);
    case 5: return go<5>(gp, nblocks, threads, smem, s, A, dt_only);
    case 6: return go<6>(gp, nblocks, threads, smem, s, A, dt_only);
    case 7: return go<7>(gp, nblocks, threads, smem, s, A, dt_only);
    default: return (int)cudaErrorInvalidValue;
  }
}

}  // namespace ftgpu
