// ft_launch.h -- host launchers of the element kernels (one translation unit per precision).
#pragma once

#include <cuda_runtime.h>

#include "ft_common.h"
#include "ft_injury.cuh"

namespace ftgpu {

// kernel<<<blocks, threads, smem, s>>>(args...), with pdl as a programmatic
// dependent of its predecessor in the stream (step_wait / step_release in
// ft_common.h).  Returns a cudaError_t value.
template <class... P, class... Args>
inline int launch_pdl(int pdl, void (*kernel)(P...), long long blocks, int threads, size_t smem,
                      cudaStream_t s, const Args &...args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)blocks);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = pdl ? 1 : 0;
  return (int)cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Launch modes of the element kernel (argument gp of launch_elem_*)
enum { kLaunchPlain = 0, kLaunchGaussPoints = 1, kLaunchInjury = 2 };

// Launch the element kernel of (etype, material) over `nblocks` patches.
// gp = kLaunchGaussPoints records per-Gauss-point F/detF/PK2, kLaunchInjury
// also updates the injury criteria of the listed elements (force pass);
// dt_only = 1 computes only the stable-time-step contribution.  Returns a
// cudaError_t value.
int launch_elem_f32(int etype, int mat, int gp, int nblocks, int threads, size_t smem,
                    cudaStream_t s, const ElemArgs<float> &A, int dt_only);
int launch_elem_f64(int etype, int mat, int gp, int nblocks, int threads, size_t smem,
                    cudaStream_t s, const ElemArgs<double> &A, int dt_only);

// Element strain pass (k_elem_strain) of one group: Voigt Green strain per
// element into Eout (group order).  Returns a cudaError_t value.
int launch_strain_f32(int etype, int nblocks, int threads, size_t smem, cudaStream_t s,
                      const ElemArgs<float> &A, double *Eout);
int launch_strain_f64(int etype, int nblocks, int threads, size_t smem, cudaStream_t s,
                      const ElemArgs<double> &A, double *Eout);
template <class R>
inline int launch_strain(int etype, int nblocks, int threads, size_t smem, cudaStream_t s,
                         const ElemArgs<R> &A, double *Eout);
template <>
inline int launch_strain<float>(int etype, int nblocks, int threads, size_t smem, cudaStream_t s,
                                const ElemArgs<float> &A, double *Eout) {
  return launch_strain_f32(etype, nblocks, threads, smem, s, A, Eout);
}
template <>
inline int launch_strain<double>(int etype, int nblocks, int threads, size_t smem,
                                 cudaStream_t s, const ElemArgs<double> &A, double *Eout) {
  return launch_strain_f64(etype, nblocks, threads, smem, s, A, Eout);
}

// Setup pass of a C3D8 group that k_elem runs (k_elem_geo): the Gauss points' inverse
// reference Jacobians and determinants into geo ([nelem/32][20][32][4]).
// Returns a cudaError_t value.
int launch_geo_f32(int nblocks, cudaStream_t s, const ElemArgs<float> &A, float *geo);

// The eight-lane C3D8 pass (ft_hexgp.cuh) and its set-up table (ten values per point)
int launch_hexgp(int mat, int gp, int nblocks, int threads, size_t smem, cudaStream_t s,
                 const ElemArgs<float> &A, int pass);
int launch_hexgp(int mat, int gp, int nblocks, int threads, size_t smem, cudaStream_t s,
                 const ElemArgs<double> &A, int pass);
int launch_hexgp_geo(int nblocks, cudaStream_t s, const ElemArgs<float> &A, float *geo);
int launch_hexgp_geo(int nblocks, cudaStream_t s, const ElemArgs<double> &A, double *geo);
// its block: eight lanes per element, at most 256 threads; slot records and
// corner forces in shared memory
inline int hexgp_threads(int PE) { return PE >= 32 ? 256 : (8 * PE + 31) / 32 * 32; }
template <class R>
constexpr size_t hexgp_smem_bytes(int PE) {
  return sizeof(R) * (8 * (size_t)kMaxLocalNodes + 24 * (size_t)PE) +
         (sizeof(R) == 8 ? 12 * (size_t)PE : 0);
}

// Dynamic shared memory of one element block: node X and u records (4 values
// each) for kMaxLocalNodes slots plus NC*3 corner forces per element, or for
// C3D8 (FP32) the larger geometry of all Gauss points, or of two pairs with
// two points' history, in the same space.
template <class R>
inline size_t elem_smem_bytes_host(int etype, int mat, int PE) {
  const int NC = etype == 0 ? 8 : 4;
  const size_t hist = mat == 5 ? 18 : (mat == 7 ? 12 : 0);
  const size_t per_elem = etype == 0 ? (hist ? 40 + 2 * hist : 80) : (size_t)NC * 3;
  const size_t slot_words = etype == 0 ? 8 : 6;  // packed records (C3D8) / component arrays
  return sizeof(R) * (slot_words * (size_t)kMaxLocalNodes + per_elem * PE) +
         (etype == 0 ? elem_csr_smem_bytes(NC, PE) : 0);
}

// Dynamic shared memory of one strain block (k_elem_strain): the slot
// records only.
template <class R>
inline size_t strain_smem_bytes_host() {
  return sizeof(R) * 8 * (size_t)kMaxLocalNodes;
}

template <class R>
inline int launch_elem(int etype, int mat, int gp, int nblocks, int threads, size_t smem,
                       cudaStream_t s, const ElemArgs<R> &A, int dt_only);
template <>
inline int launch_elem<float>(int etype, int mat, int gp, int nblocks, int threads, size_t smem,
                              cudaStream_t s, const ElemArgs<float> &A, int dt_only) {
  return launch_elem_f32(etype, mat, gp, nblocks, threads, smem, s, A, dt_only);
}
template <>
inline int launch_elem<double>(int etype, int mat, int gp, int nblocks, int threads,
                               size_t smem, cudaStream_t s, const ElemArgs<double> &A,
                               int dt_only) {
  return launch_elem_f64(etype, mat, gp, nblocks, threads, smem, s, A, dt_only);
}

}  // namespace ftgpu
