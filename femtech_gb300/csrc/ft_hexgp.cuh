// ft_hexgp.cuh -- C3D8 element pass with eight lanes per element, one Gauss
// point and one corner each.  Same contract as k_elem (ft_elem.cuh): force,
// stress update, stable-dt contribution, injury criteria and in-block
// deterministic assembly of one patch per block.
//
// Where it is used and why:
//  * FP64, always.  This GPU issues one FP64 warp instruction per SM in 16
//    cycles, so the pass is bound by the count of FP64 instructions and by how
//    evenly they spread over the SMs; everything else (shuffles, selects,
//    loads) is hidden.  One thread per element held eight Gauss points in a
//    serial loop, spilled, and left a 1,000-element mesh on 8 SMs.
//  * FP32 for small meshes, where a step waits for one warp's serial chain of
//    eight Gauss points; the larger ones are bound by issue slots, of which
//    the shuffles here take more.
//
// The trilinear element's transforms run as butterflies over the element's
// eight lanes (bit 0: xi, bit 1: eta, bit 2: zeta; lane bits (bx, by, bz) hold
// corner (2 bx - 1, 2 by - 1, 2 bz - 1), then pattern xi^bx eta^by zeta^bz,
// then Gauss point of those signs): a stage is one operation per value, and
// corners -> patterns -> Gauss points takes 9 + 18 per lane.  The transposed
// way back (Gauss points -> moments -> corners) takes 30 + 9.
// Measured (element pass, one thread per element -> eight lanes): FP64
// 1,000 Neo-Hookean 159 -> 22 us, 32,000 Ogden 1,004 -> 239 us (with the laws'
// series, ft_materials.cuh; 195 us with the step bounds); FP32 3,927 Ogden 18.9 -> 8.5 us.
// Geometry: A^{-1} / 8 and det A of every Gauss point from a set-up table
// [8 nelem/32][10][32] (the 1/8 of both transforms, exact).
#pragma once

#include "ft_elem.cuh"
#include "ft_launch.h"

namespace ftgpu {

constexpr int kHexGpThreads = 256;  // largest block: 32 elements at a time

template <class R>
__device__ __forceinline__ R shx(R v, int mask) {
  return __shfl_xor_sync(0xffffffffu, v, mask);
}
__device__ __forceinline__ float flip_if(float x, bool f) { return f ? -x : x; }
__device__ __forceinline__ double flip_if(double x, bool f) {
  return __hiloint2double(__double2hiint(x) ^ (f ? (int)0x80000000u : 0), __double2loint(x));
}
// one butterfly stage, signs -> patterns: sum on lane bit 0, (+) - (-) on bit 1
template <class R>
__device__ __forceinline__ R had(R v, int mask, bool bit) {
  return v + flip_if(shx(v, mask), bit);
}
// patterns -> values at -c (lane bit 0) and +c (bit 1): A -+ c B, A the value
// of the lane with bit 0 and B of its partner; cs = -c or +c of this lane
template <class R>
__device__ __forceinline__ R ev(R v, int mask, bool bit, R cs) {
  const R o = shx(v, mask);
  return (bit ? o : v) + cs * (bit ? v : o);
}

template <class R> struct UBits;
template <> struct UBits<float> { typedef unsigned T; };
template <> struct UBits<double> { typedef unsigned long long T; };
__device__ __forceinline__ unsigned ubits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ unsigned long long ubits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}
__device__ __forceinline__ float from_ubits(unsigned b) { return __uint_as_float(b); }
__device__ __forceinline__ double from_ubits(unsigned long long b) {
  return __longlong_as_double((long long)b);
}
// J is not above zero, or is NaN (J = 1 + (J - 1): never subnormal)
__device__ __forceinline__ bool bad_j(float J) { return !(J > 0.f); }
__device__ __forceinline__ bool bad_j(double J) {
  const int hi = __double2hiint(J);
  return hi <= 0 || hi > 0x7ff00000;
}
__device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }
__device__ __forceinline__ bool is_zero(double x) {
  return ((unsigned long long)__double_as_longlong(x) << 1) == 0ull;
}

// The element's stable step l / c, l = volume / largest face area of the
// current geometry (CalculateCharacteristicLength_C3D8.cpp:6-29, the face rule
// of Geometry.cpp:29-64 with its signed parallelogram test), from the lane's
// current corner y and vol, its share of the volume (SHARE) or the volume.  A lane takes the three
// faces that meet in its corner, and on each the quadrature point next to it:
// the face's tangents there are butterflies of the patterns (+-1 on the face's
// axis, +-1/sqrt 3 or, for a parallelogram, 0 on the others).  All values in
// units of 8 x the patterns.  Same on all eight lanes.
template <class R>
__device__ __forceinline__ R hexgp_volume(R detJ) {
  detJ += shx(detJ, 1);
  detJ += shx(detJ, 2);
  return detJ + shx(detJ, 4);
}
template <bool SHARE, class R>
__device__ __forceinline__ R hexgp_dt(const R (&y)[3], R vol, const MatP<R> &mp, bool bx, bool by,
                                      bool bz) {
  R h[3], w1[3], w2[3], w4[3];
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    h[d] = had(had(had(y[d], 1, bx), 2, by), 4, bz);
    w1[d] = __shfl_sync(0xffffffffu, h[d], lane | 1);  // patterns with xi
    w2[d] = __shfl_sync(0xffffffffu, h[d], lane | 2);  // with eta
    w4[d] = __shfl_sync(0xffffffffu, h[d], lane | 4);  // with zeta
  }
  const R ox = bx ? R(1) : R(-1), oy = by ? R(1) : R(-1), oz = bz ? R(1) : R(-1);
  constexpr double t = 0.57735026918962576451;
  // area of the face with axis mask m0 at its lane bit b0, tangents from p
  // (patterns along axis A) and q (along axis B), in-face masks mA, mB
  auto face = [&](const R (&p)[3], const R (&q)[3], int m0, bool b0, R o0, int mA, bool bA, R oA,
                  int mB, bool bB, R oB) {
    R a[3], b[3], cD[3];
    bool flat = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a[d] = ev(p[d], m0, b0, o0);  // lanes bB = 0: c1; bB = 1: the twist cD
      b[d] = ev(q[d], m0, b0, o0);  // lanes bA = 0: c2; bA = 1: cD
      const R x = shx(a[d], mB);
      cD[d] = bB ? a[d] : x;
      flat = flat && below_pos(cD[d], R(8e-6));
      a[d] = bB ? x : a[d];
      const R z = shx(b[d], mA);
      b[d] = bA ? z : b[d];
    }
    const R kA = flat ? R(0) : R(t) * oB, kB = flat ? R(0) : R(t) * oA;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a[d] += kA * cD[d];
      b[d] += kB * cD[d];
    }
    const R nx = a[1] * b[2] - a[2] * b[1], ny = a[2] * b[0] - a[0] * b[2],
            nz = a[0] * b[1] - a[1] * b[0];
    R s = d_sqrt(nx * nx + ny * ny + nz * nz);
    s += shx(s, mA);
    return s + shx(s, mB);
  };
  // (areas are not negative: compared as bits)
  typename UBits<R>::T am = ubits(face(w1, w2, 4, bz, oz, 1, bx, ox, 2, by, oy));
  const auto a2 = ubits(face(w1, w4, 2, by, oy, 1, bx, ox, 4, bz, oz)),
             a3 = ubits(face(w2, w4, 1, bx, ox, 2, by, oy, 4, bz, oz));
  am = a2 > am ? a2 : am;
  am = a3 > am ? a3 : am;
#pragma unroll
  for (int m = 1; m <= 4; m <<= 1) {
    const auto o = __shfl_xor_sync(0xffffffffu, am, m);
    am = o > am ? o : am;
  }
  if (SHARE) vol = hexgp_volume(vol);
  if constexpr (sizeof(R) == 4) return R(64) * vol / from_ubits(am) * mp.inv_ce;
  return R(64) * vol / (from_ubits(am) * R(mp.ce));
}

// Bounds of the same step for FP64, in FP32: only the elements whose lower
// bound is not above the block's least upper one (nor above the minimum so far)
// take hexgp_dt, a quarter to a third of the pass' FP64 operations, on a pipe that issues one
// warp instruction in 16 cycles (32,000 Ogden elements 245 -> 201 us a step,
// 42,000 of material 7 362 -> 305; 86 % of the pipe then).  r: the current corner relative to the
// element's first one; vol: the volume (FP64, rounded).  The arithmetic is
// hexgp_dt's.  Errors, with eps = 2^-24 and Rm the largest |r|: the patterns
// carry at most 32 eps Rm (inputs and three sums of up to 8 Rm), the face's
// tangents 160 eps Rm, so a point's area sqrt 3 160 eps Rm (|a| + |b|) and the
// face's sum four times that; 1200 takes in the roundings of the product, the
// root and the sums.  A twist within its own error of the parallelogram test,
// values outside FP32's comfortable range and NaNs leave the element undecided:
// lo = 0, hi = inf.
__device__ __forceinline__ void hexgp_dt_bounds(const float (&r)[3], float vol, float inv_ce, bool bx,
                                                bool by, bool bz, float &lo, float &hi) {
  constexpr float kEps = 1.f / 16777216.f;
  const float inf = r_inf<float>();
  const int lane = threadIdx.x & 31;
  float rm = fmaxf(fmaxf(fabsf(r[0]), fabsf(r[1])), fabsf(r[2]));
#pragma unroll
  for (int m = 1; m <= 4; m <<= 1) rm = fmaxf(rm, shx(rm, m));
  float h[3], w1[3], w2[3], w4[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    h[d] = had(had(had(r[d], 1, bx), 2, by), 4, bz);
    w1[d] = __shfl_sync(0xffffffffu, h[d], lane | 1);
    w2[d] = __shfl_sync(0xffffffffu, h[d], lane | 2);
    w4[d] = __shfl_sync(0xffffffffu, h[d], lane | 4);
  }
  const float ox = bx ? 1.f : -1.f, oy = by ? 1.f : -1.f, oz = bz ? 1.f : -1.f;
  const float t = 0.57735026918962576451f, tol = 8e-6f, dtw = 100.f * kEps * rm;
  float size = rm >= 1e-8f && rm <= 1e8f ? 0.f : inf;  // largest |a| + |b|
  auto face = [&](const float (&p)[3], const float (&q)[3], int m0, bool b0, float o0, int mA,
                  bool bA, float oA, int mB, bool bB, float oB) {
    float a[3], b[3], cD[3];
    bool flat = true, open = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a[d] = ev(p[d], m0, b0, o0);
      b[d] = ev(q[d], m0, b0, o0);
      const float x = shx(a[d], mB);
      cD[d] = bB ? a[d] : x;
      flat = flat && cD[d] < tol;
      open = open || !(fabsf(cD[d] - tol) > dtw);
      a[d] = bB ? x : a[d];
      const float z = shx(b[d], mA);
      b[d] = bA ? z : b[d];
    }
    const float kA = flat ? 0.f : t * oB, kB = flat ? 0.f : t * oA;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a[d] += kA * cD[d];
      b[d] += kB * cD[d];
    }
    const float nx = a[1] * b[2] - a[2] * b[1], ny = a[2] * b[0] - a[0] * b[2],
                nz = a[0] * b[1] - a[1] * b[0];
    size = fmaxf(size, open ? inf
                            : (fabsf(a[0]) + fabsf(a[1]) + fabsf(a[2])) +
                                  (fabsf(b[0]) + fabsf(b[1]) + fabsf(b[2])));
    float s = sqrtf(nx * nx + ny * ny + nz * nz);
    s += shx(s, mA);
    return s + shx(s, mB);
  };
  float am = face(w1, w2, 4, bz, oz, 1, bx, ox, 2, by, oy);
  am = fmaxf(am, face(w1, w4, 2, by, oy, 1, bx, ox, 4, bz, oz));
  am = fmaxf(am, face(w2, w4, 1, bx, ox, 2, by, oy, 4, bz, oz));
#pragma unroll
  for (int m = 1; m <= 4; m <<= 1) {
    am = fmaxf(am, shx(am, m));
    size = fmaxf(size, shx(size, m));
  }
  const float err = 1200.f * kEps * rm * size;
  const float v = 64.f * vol * inv_ce;
  const float l = v / (am + err) * (1.f - 1e-6f), u = v / (am - err) * (1.f + 1e-6f);
  lo = l > 1e-30f && l < 1e30f ? l : 0.f;
  hi = am > err && u > 1e-30f && u < 1e30f ? u : inf;
}

// FP64: at most 128 registers (two blocks per SM, 16 warps); the pipe takes
// one instruction in 16 cycles, so more warps would not help.  FP32: the small
// meshes it serves put one block on an SM.
// BOUND: stable steps by hexgp_dt_bounds first (FP64 force passes).
template <class R, int MAT, bool GP, bool INJ, bool BOUND = false>
__global__ void __launch_bounds__(kHexGpThreads, 2) k_hexgp(const ElemArgs<R> A, int pass) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Slot4<R> *shX = reinterpret_cast<Slot4<R> *>(smem_raw);
  Slot4<R> *shU = shX + kMaxLocalNodes;
  R *shF = reinterpret_cast<R *>(shU + kMaxLocalNodes);  // [element][corner][3]
  const int T = blockDim.x, t = threadIdx.x, lane = t & 31;
  const int p = A.patch_begin + blockIdx.x;
  const int inst = A.patch_inst[p];
  const int e0 = A.patch_elem_off[p], ne = A.patch_elem_off[p + 1] - e0;
  const int s0 = A.patch_node_off[p], ns = A.patch_node_off[p + 1] - s0;
  const Clock *ck = A.clock + A.parity * A.ninst + inst;
  for (int i = t; i < ns; i += T) {
    cp_async_small<sizeof(R)>(&shX[i].x, A.sX + s0 + i);
    cp_async_small<sizeof(R)>(&shX[i].y, A.sX + A.S + s0 + i);
    cp_async_small<sizeof(R)>(&shX[i].z, A.sX + 2 * A.S + s0 + i);
  }
  step_wait();  // the displacements and the clock are the node pass'
  step_release();
  for (int i = t; i < ns; i += T) {
    const R *us = A.sU + 4ll * (s0 + i);
#pragma unroll
    for (int h = 0; h < (int)sizeof(Slot4<R>) / 16; ++h)
      cp_async16(reinterpret_cast<char *>(shU + i) + 16 * h, us + h * (16 / sizeof(R)));
  }
  // lane l of the element: bits, corner and Gauss point of these signs
  const int l8 = t & 7;
  const bool bx = l8 & 1, by = l8 & 2, bz = l8 & 4;
  // the elements' step bounds and volumes (BOUND)
  R *shVol = shF + 24 * ne;
  float *shLo = reinterpret_cast<float *>(shVol + ne);
  __shared__ unsigned cut;  // least upper bound, as bits
  if (BOUND && t == 0) cut = ubits(r_inf<float>());
  const int corner = (bz ? 4 : 0) + (by ? (bx ? 2 : 3) : (bx ? 1 : 0));
  const int gp = (bz ? 0 : 4) + (by ? (bx ? 2 : 3) : (bx ? 1 : 0));
  const R c = R(0.577350269189626);
  const R cx = bx ? c : -c, cy = by ? c : -c, cz = bz ? c : -c;
  const int bits = __popc(l8);
  const R cp = bits < 2 ? R(1) : (bits == 2 ? c : c * c);
  cp_async_wait_all();
  if (A.use_clock && ck->done) return;  // past its end time: the whole block
  const R dt = A.use_clock ? R(ck->dt) : R(A.dt_direct);
  __syncthreads();
  typename UBits<R>::T dmin = ubits(r_inf<R>());
  int bad = 0;
  R iv[4] = {-r_inf<R>(), r_inf<R>(), -r_inf<R>(), -r_inf<R>()};
  int ij[4] = {0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff}, ic[4] = {-1, -1, -1, -1};
  // T / 8 elements at a time; every warp takes part in the shuffles as a whole
  for (int i0 = 0; i0 < ne; i0 += T >> 3) {
    const int i = i0 + (t >> 3);
    const bool act = i < ne;
    const int e = e0 + (act ? i : 0);
    const long long el = e - A.elem_begin, sg = 8 * el + l8;
    const R *geo = A.geo + blk_at(sg, 10);
    R Q[3][3];
#pragma unroll
    for (int k = 0; k < 9; ++k) Q[k / 3][k % 3] = geo[k * kLaneBlk];
    const R detA = geo[9 * kLaneBlk];
    int ln = A.lconn[8 * el + corner];
    const int pw = A.epid[e];
    if (ln >= ns) {
      bad |= 2;
      ln = 0;
    }
    const Slot4<R> us = shU[ln], xs = shX[ln];
    const R u[3] = {us.x, us.y, us.z};
    const MatP<R> &mp = A.mats[pw & 0x7fffffff];
    R a0[3] = {R(1), R(0), R(0)};
    if (MAT == 7) {
      a0[0] = A.fib[e];
      a0[1] = A.fib[A.E + e];
      a0[2] = A.fib[2 * A.E + e];
    }
    // displacement patterns, then H[d][i] = du_d / dxi_i at the Gauss point (x 8)
    R H[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const R h = had(had(had(u[d], 1, bx), 2, by), 4, bz);
      const R h1 = __shfl_sync(0xffffffffu, h, lane | 1), h2 = __shfl_sync(0xffffffffu, h, lane | 2),
              h4 = __shfl_sync(0xffffffffu, h, lane | 4);
      H[d][0] = ev(ev(h1, 2, by, cy), 4, bz, cz);
      H[d][1] = ev(ev(h2, 1, bx, cx), 4, bz, cz);
      H[d][2] = ev(ev(h4, 1, bx, cx), 2, by, cy);
    }
    R D[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        D[r][j] = H[r][0] * Q[j][0] + H[r][1] * Q[j][1] + H[r][2] * Q[j][2];
    const R Jm1 = jm1_of(D);
    const R J = 1 + Jm1;
    if (MAT == 7 && pass == kPassSurrogateFeatures) {
      if (act) {
        if (bad_j(J) || is_zero(detA)) bad |= 1;
        write_surrogate_features(D, a0, A.law, A.surr_x + (8 * el + gp) * kMlpIn);
      }
      continue;
    }
    {
      const R y[3] = {xs.x + u[0], xs.y + u[1], xs.z + u[2]};
      if constexpr (BOUND) {
        const R vol = hexgp_volume(J * detA);
        float r[3], lo, hi;
#pragma unroll
        for (int d = 0; d < 3; ++d)
          r[d] = d2f_bits(y[d] - __shfl_sync(0xffffffffu, y[d], lane & 24));
        hexgp_dt_bounds(r, d2f_bits(vol), d2f_bits(mp.inv_ce), bx, by, bz, lo, hi);
        if (act && l8 == 0) {
          shVol[i] = vol;
          shLo[i] = pw >= 0 ? lo : r_inf<float>();
          if (pw >= 0) atomicMin(&cut, ubits(hi));
        }
      } else {
        const auto b = ubits(hexgp_dt<true>(y, J * detA, mp, bx, by, bz));
        if (act && pw >= 0 && b < dmin) dmin = b;
      }
    }
    if (pass == kPassDt) continue;
    if (act && (bad_j(J) || is_zero(detA))) bad |= 1;
    if (INJ) {  // the listed element's averaged Green strain
      const Sym6<R> M = two_E(D);
      R Es[6] = {M.xx, M.yy, M.zz, M.yz, M.xz, M.xy};
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        Es[k] += shx(Es[k], 1);
        Es[k] += shx(Es[k], 2);
        Es[k] = R(0.0625) * (Es[k] + shx(Es[k], 4));
      }
      const int ci = act && l8 == 0 ? A.inj_cidx[e] : -1;
      R v[4] = {0, 0, 0, 0};
      bool above[2] = {false, false};
      if (ci >= 0) {
        int vj[4], vc[4];
        injury_element<R>(A, ci, Es, dt, v, vj, vc, above);
        injury_take<R>(v, vj, vc, iv, ij, ic);
      }
      injury_append<R>(A, 0, above[0], v[0]);
      injury_append<R>(A, 1, above[1], v[3]);
    }
    R G[3][3];
    {
      R pc[4];
      prony_consts<R, MAT>(mp, dt, pc);
      const float *sy = (MAT == 7 && A.surr_y) ? A.surr_y + (8 * el + gp) * kMlpOut : nullptr;
      R *hist = hist_comps(MAT) > 0 ? A.hist + blk_at(sg, hist_comps(MAT)) : nullptr;
      Sym6<R> S;
      if ((MAT == 5 || MAT == 7) && !act)  // (its history is another element's)
        S = Sym6<R>{0, 0, 0, 0, 0, 0};
      else
        S = stress_at<R, MAT>(mp, D, Jm1, a0, hist, pc, sy, A.law, HistGlobal<R>{hist},
                              PartAt<R>{&mp});
      if (GP && act) {
        const long long q = A.gpbase + 8 * el + gp;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int j = 0; j < 3; ++j) A.gpF[9 * q + r + 3 * j] = double((r == j ? R(1) : R(0)) + D[r][j]);
        A.gpJ[q] = double(J);
        A.gpS[6 * q + 0] = S.xx;
        A.gpS[6 * q + 1] = S.yy;
        A.gpS[6 * q + 2] = S.zz;
        A.gpS[6 * q + 3] = S.yz;
        A.gpS[6 * q + 4] = S.xz;
        A.gpS[6 * q + 5] = S.xy;
      }
      // w det J B0^T S with w = 1: P = det A (S + D S), G = P A^{-1} (/ 8)
      const R sxx = detA * S.xx, syy = detA * S.yy, szz = detA * S.zz, syz = detA * S.yz,
              sxz = detA * S.xz, sxy = detA * S.xy;
      const R s[3][3] = {{sxx, sxy, sxz}, {sxy, syy, syz}, {sxz, syz, szz}};
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        R P[3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
          P[j] = s[r][j] + D[r][0] * s[0][j] + D[r][1] * s[1][j] + D[r][2] * s[2][j];
#pragma unroll
        for (int j = 0; j < 3; ++j) G[r][j] = P[0] * Q[0][j] + P[1] * Q[1][j] + P[2] * Q[2][j];
      }
    }
    // moments of the eight Gauss points: pattern p collects c^(|p| - 1) times
    // the transform of column i under pattern p - i, for each axis i in p
    // (columns 1 and 2 share their last stage), then the corners
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      R g0 = had(G[d][0], 4, bz), g1 = had(G[d][1], 4, bz), g2 = G[d][2] + shx(G[d][2], 4);
      g0 = had(g0, 2, by);
      g2 = had(g2, 2, by);
      g1 = g1 + shx(g1, 2);
      g1 = (by ? g1 : R(0)) + (bz ? g2 : R(0));
      g1 = had(g1, 1, bx);
      g0 = g0 + shx(g0, 1);
      R m = cp * (g1 + (bx ? g0 : R(0)));
      m = m + flip_if(shx(m, 1), !bx);
      m = m + flip_if(shx(m, 2), !by);
      m = m + flip_if(shx(m, 4), !bz);
      if (act) shF[24 * i + 3 * corner + d] = m;
    }
  }
  if (bad) atomicOr(A.err, (bad & 1 ? kErrInverted : 0) | (bad & 2 ? kErrIndex : 0));
  if (pass == kPassSurrogateFeatures) return;  // features only (uniform per block)
  if (INJ && pass == kPassForce)
    injury_block_extremes<kHexGpThreads>(iv, ij, ic, reinterpret_cast<InjuryPart *>(A.inj_part) + p);
  if constexpr (BOUND) {
    // the exact steps of the elements that the bounds leave
    __syncthreads();
    unsigned long long *gmin = A.dtmin + A.parity * A.ninst + inst;
    const float cutf = from_ubits(cut);
    const unsigned long long seen = *reinterpret_cast<volatile unsigned long long *>(gmin);
    for (int i0 = 0; i0 < ne; i0 += T >> 3) {
      const int i = i0 + (t >> 3);
      const float lo = i < ne ? shLo[i] : r_inf<float>();
      const bool mine = lo <= cutf && lo < r_inf<float>() && ubits(f2d_bits(lo)) <= seen;
      if (!__any_sync(0xffffffffu, mine)) continue;
      const int e = e0 + (i < ne ? i : 0);
      int ln = A.lconn[8ll * (e - A.elem_begin) + corner];
      if (ln >= ns) ln = 0;
      const Slot4<R> us = shU[ln], xs = shX[ln];
      const R y[3] = {xs.x + us.x, xs.y + us.y, xs.z + us.z};
      const auto b = ubits(hexgp_dt<false>(y, mine ? shVol[i] : R(1),
                                           A.mats[A.epid[e] & 0x7fffffff], bx, by, bz));
      if (mine && b < dmin) dmin = b;
    }
  }
  // block minimum of the time steps as bits (positive values order like them;
  // a negative or NaN step of an inverted element is larger than any)
#pragma unroll
  for (int m = 8; m <= 16; m <<= 1) {  // (the eight lanes of an element agree)
    const auto o = __shfl_xor_sync(0xffffffffu, dmin, m);
    dmin = o < dmin ? o : dmin;
  }
  __shared__ typename UBits<R>::T wmin[kHexGpThreads / 32];
  if (lane == 0) wmin[t >> 5] = dmin;
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < (T + 31) / 32; ++w) dmin = wmin[w] < dmin ? wmin[w] : dmin;
    atomicMin(A.dtmin + A.parity * A.ninst + inst,
              (unsigned long long)__double_as_longlong(double(from_ubits(dmin))));
  }
  if (pass != kPassForce) return;
  // in-block assembly: local node i sums its corners in (element, corner) order
  const uint16_t *lp = A.lptr + s0 + p, *le = A.lent + A.patch_ent_off[p];
  for (int i = t; i < ns; i += T) {
    const int b = lp[i], en = lp[i + 1];
    R f0 = 0, f1 = 0, f2 = 0;
    for (int k = b; k < en; ++k) {
      const R *f = shF + 3 * (int)le[k];
      f0 += f[0];
      f1 += f[1];
      f2 += f[2];
    }
    reinterpret_cast<Slot4<R> *>(A.sF)[s0 + i] = Slot4<R>{f0, f1, f2, R(0)};
  }
}

// Set-up pass of a group that k_hexgp runs: A^{-1} / 8 (row major) and det A
// of the reference geometry at each Gauss point (ShapeFunction_C3D8.cpp:35-120),
// in FP64 from the slot coordinates, as [8 nelem/32][10][32] of points 8
// element + lane.
template <class R>
__global__ void __launch_bounds__(kHexGpThreads) k_hexgp_geo(const ElemArgs<R> A, R *geo) {
  __shared__ double shX[3][kMaxLocalNodes];
  const int p = A.patch_begin + blockIdx.x;
  const int e0 = A.patch_elem_off[p], ne = A.patch_elem_off[p + 1] - e0;
  const int s0 = A.patch_node_off[p], ns = A.patch_node_off[p + 1] - s0;
  for (int i = threadIdx.x; i < ns && i < kMaxLocalNodes; i += blockDim.x)
#pragma unroll
    for (int d = 0; d < 3; ++d) shX[d][i] = double(A.sX[d * A.S + s0 + i]);
  __syncthreads();
  int bad = 0;
  for (int q = threadIdx.x; q < 8 * ne; q += blockDim.x) {
    const long long el = e0 + (q >> 3) - A.elem_begin;
    const int l8 = q & 7;
    double x[8][3];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      int l = A.lconn[8 * el + a];
      if (l >= ns || l >= kMaxLocalNodes) {
        bad |= kErrIndex;
        l = 0;
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) x[a][d] = shX[d][l];
    }
    double hx[7][3];
    hex_hadamard(x, hx);
    const double c = 0.577350269189626;
    const double xi = l8 & 1 ? c : -c, et = l8 & 2 ? c : -c, ze = l8 & 4 ? c : -c;
    const double ez = et * ze, xz = xi * ze, xe = xi * et;
    double Am[3][3], Ad[3][3], det;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      Am[0][d] = hx[0][d] + et * hx[3][d] + ze * hx[4][d] + ez * hx[6][d];
      Am[1][d] = hx[1][d] + xi * hx[3][d] + ze * hx[5][d] + xz * hx[6][d];
      Am[2][d] = hx[2][d] + xi * hx[4][d] + et * hx[5][d] + xe * hx[6][d];
    }
    adj3(Am, Ad, det);
    const double id = 0.125 / det;  // det = 0: non-finite entries, flagged by the force pass
#pragma unroll
    for (int k = 0; k < 10; ++k) geo[blk_at(8 * el + l8, 10) + k * kLaneBlk] = R(k < 9 ? Ad[k / 3][k % 3] * id : det);
  }
  if (bad) atomicOr(A.err, bad);
}

// The launches ask for no more than the default 48 KB: the largest patches of
// each precision with the kernels' own static arrays (the injury extremes',
// the block minima and the bounds' cut: 576 bytes)
constexpr size_t kHexGpStatic = 1024;
static_assert(hexgp_smem_bytes<double>(128) + kHexGpStatic <= 48 * 1024,
              "an FP64 patch of 128 elements fits the default shared memory");
static_assert(hexgp_smem_bytes<float>(kMaxPatchElems) + kHexGpStatic <= 48 * 1024,
              "the largest FP32 patch fits the default shared memory");

// The launcher of one precision's instantiations (ft_hexgp_f32.cu, _f64.cu)
template <class R, int MAT>
int hexgp_go(int gp, int nb, int th, size_t sm, cudaStream_t s, const ElemArgs<R> &A, int pass) {
  if (gp == kLaunchGaussPoints)
    return launch_pdl(A.pdl, k_hexgp<R, MAT, true, false>, nb, th, sm, s, A, pass);
  if (gp == kLaunchInjury)
    return launch_pdl(A.pdl, k_hexgp<R, MAT, false, true>, nb, th, sm, s, A, pass);
  if constexpr (sizeof(R) == 8)
    if (A.dt_bounds)
      return launch_pdl(A.pdl, k_hexgp<R, MAT, false, false, true>, nb, th, sm, s, A, pass);
  return launch_pdl(A.pdl, k_hexgp<R, MAT, false, false>, nb, th, sm, s, A, pass);
}

template <class R>
int hexgp_by_mat(int mat, int gp, int nb, int th, size_t sm, cudaStream_t s, const ElemArgs<R> &A,
                 int pass) {
  switch (mat) {
    case 0: return hexgp_go<R, 0>(gp, nb, th, sm, s, A, pass);
    case 1: return hexgp_go<R, 1>(gp, nb, th, sm, s, A, pass);
    case 2: return hexgp_go<R, 2>(gp, nb, th, sm, s, A, pass);
    case 3: return hexgp_go<R, 3>(gp, nb, th, sm, s, A, pass);
    case 4: return hexgp_go<R, 4>(gp, nb, th, sm, s, A, pass);
    case 5: return hexgp_go<R, 5>(gp, nb, th, sm, s, A, pass);
    case 6: return hexgp_go<R, 6>(gp, nb, th, sm, s, A, pass);
    case 7: return hexgp_go<R, 7>(gp, nb, th, sm, s, A, pass);
    default: return (int)cudaErrorInvalidValue;
  }
}

}  // namespace ftgpu
