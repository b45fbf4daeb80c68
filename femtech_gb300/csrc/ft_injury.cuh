// ft_injury.cuh -- per-step injury criteria of the brain drivers on the GPU
// (examples/ex5/ex5.cpp:1311-1430, CalculateInjuryCriterions): principal
// strains of the listed elements, running extremes, sticky threshold flags and
// the largest 95th percentiles of MPS and of MPS x strain rate.
//
// Only a step whose percentile exceeds the running maximum changes anything,
// and then the percentile is one of the values above that maximum.  So the
// force pass, which forms the values, appends those above it to a candidate
// list (some 5 % of the elements while a percentile grows, none while it does
// not, all at a run's first step), and one launch ends the step:
// k_injury_select takes the percentile's rank among the candidates by an exact
// radix selection, a cluster of eight blocks per selection, and the extremes
// from the patches' partials.  The
// elements' list flags follow in the next force pass, which has the step's
// values at hand (k_injury_out applies them when they are read).
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "ft_common.h"

namespace ftgpu {

// running state (FP64 values; element ids are the reference's)
struct InjuryState {
  double max_strain, max_strain_time, min_strain, min_strain_time;
  double max_shear, max_shear_time, max_psxsr, max_psxsr_time;
  int max_strain_elem, min_strain_elem, max_shear_elem, max_psxsr_elem;
  double mps95, mps95_time, mpsxsr95, mpsxsr95_time;
  int mps95_count, mpsxsr95_count;
  long long steps;
};

// flags per injury element (bits)
enum { kInjMps15 = 1, kInjMps30 = 2, kInjPsr120 = 4, kInjPsxsr28 = 8, kInjInMps95 = 16,
       kInjInMpsxsr95 = 32 };

// per-block partial extremes of one step: value, the caller's list position
// (tie-break) and the compact index of the element
struct InjuryPart {
  double v[4];  // max strain, min strain, max shear, max psxsr
  int j[4];     // list position
  int c[4];     // compact index
};

// The running maxima of the two percentiles as the force pass compares with
// them, and the last step's update: upd[sel] set when it took a new maximum v
// (both also in FP32, exactly: they are values of the element precision)
struct InjuryRun {
  double run[2], v[2];
  float runf[2], vf[2];
  int upd[2];
  unsigned count[2][32];  // candidates of the step ([sel][0]; a line each)
};
template <class R> __device__ __forceinline__ R inj_run(const InjuryRun *q, int sel);
template <> __device__ __forceinline__ float inj_run<float>(const InjuryRun *q, int sel) { return q->runf[sel]; }
template <> __device__ __forceinline__ double inj_run<double>(const InjuryRun *q, int sel) { return q->run[sel]; }
template <class R> __device__ __forceinline__ R inj_thr(const InjuryRun *q, int sel);
template <> __device__ __forceinline__ float inj_thr<float>(const InjuryRun *q, int sel) { return q->vf[sel]; }
template <> __device__ __forceinline__ double inj_thr<double>(const InjuryRun *q, int sel) { return q->v[sel]; }

constexpr int kInjThreads = 512;
constexpr int kInjCluster = 8;            // blocks per selection
constexpr int kInjSelectSmem = 96 << 10;  // a block's candidate keys on the chip

// The listed elements are kept in group order ("compact" index c): element e
// (group order) is listed when cidx[e] >= 0; upos[c] is its position in the
// caller's list (ties go to the smaller position, as in the reference's loop)
// and eref[c] its reference id.
template <class R>
struct InjuryArgs {
  const int *eref;       // [n]
  const R *cand;         // [2][n] the step's candidates
  const InjuryPart *part;  // [patches] block extremes of the step
  InjuryRun *run;
  InjuryState *state;
  const Clock *clock;    // clock[0] of the step (single instance)
  int n, parity, npart;
};

// principal strains of the symmetric strain in the trigonometric form of
// CalculateStrain.cpp:38-74
template <class T>
__device__ __forceinline__ void principal_strains(T xx, T yy, T zz, T yz, T xz, T xy, T &mx,
                                                  T &mn, T &sh) {
  const T a = xx, b = xy, c = xz, d = yy, e = yz, f = zz;
  const T p1 = b * b + c * c + e * e;
  T e1, e2, e3;
  if (p1 == T(0)) {
    e1 = a;
    e2 = d;
    e3 = f;
  } else {
    T I1 = a + d + f;
    const T I2 = a * (d + f) + d * f - b * b - c * c - e * e;
    const T I3 = a * d * f + T(2) * b * c * e - b * b * f - c * c * d - e * e * a;
    const T Q = (T(3) * I2 - I1 * I1) / T(9);
    const T Rr = (T(2) * I1 * I1 * I1 - T(9) * I1 * I2 + T(27) * I3) / T(54);
    const T theta = acos(Rr / sqrt(-Q * Q * Q));
    const T sq = T(2) * sqrt(-Q);
    const T kPi = T(3.141592653589793);
    I1 = I1 / T(3);
    e1 = sq * cos(theta / T(3)) + I1;
    e2 = sq * cos((theta + T(2) * kPi) / T(3)) + I1;
    e3 = sq * cos((theta + T(4) * kPi) / T(3)) + I1;
  }
  const T hi = fmax(e3, fmax(e2, e1)), lo = fmin(e3, fmin(e2, e1));
  sh = T(0.5) * (hi - lo);
  mx = hi > T(0) ? hi : T(0);
  mn = lo < T(0) ? lo : T(0);
}

// order-preserving unsigned keys of floating-point values
__device__ __forceinline__ uint32_t fkey(float x) {
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
__device__ __forceinline__ uint64_t fkey(double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double fkey_inv(uint64_t k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

// better (value, list index) of two candidates for extreme k (k = 1 is a
// minimum): the better value, then the smaller list index
template <class V>
__device__ __forceinline__ bool inj_better(int k, V bv, int bj, V av, int aj) {
  return (k == 1) ? (bv < av || (bv == av && bj < aj)) : (bv > av || (bv == av && bj < aj));
}

// The list flags of an element after the last step's update
template <class R>
__device__ __forceinline__ uint8_t inj_list_flags(const InjuryRun *q, uint8_t f, R ps, R psxsr) {
  if (q->upd[0])
    f = ps >= inj_thr<R>(q, 0) ? (f | kInjInMps95) : (f & (uint8_t)~kInjInMps95);
  if (q->upd[1])
    f = psxsr >= inj_thr<R>(q, 1) ? (f | kInjInMpsxsr95) : (f & (uint8_t)~kInjInMpsxsr95);
  return f;
}

// The value of rank k = (int)(0.95 n) - 1 (rank 0 if negative) of a selection,
// when it exceeds the running maximum: the n - count values at or below the
// maximum come before every candidate.  Eight bits per pass over the
// candidates' keys, each block of the cluster on its share; lanes with the
// same bin add once (the strains of one tissue share their top bits), and
// every block sums the eight histograms through distributed shared memory, so
// one cluster barrier per pass suffices (the other buffer is cleared
// meanwhile: its readers passed the barrier before).
template <class R>
__device__ __forceinline__ void injury_select(const InjuryArgs<R> &A, int sel, double time,
                                              unsigned char *sm) {
  typedef typename std::conditional<sizeof(R) == 8, uint64_t, uint32_t>::type K;
  constexpr int KB = sizeof(K) * 8;
  __shared__ unsigned hist[2][256], total[256];
  __shared__ unsigned s_digit, s_below;
  const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int t = threadIdx.x, lane = t & 31;
  const unsigned rank = cl.block_rank();
  InjuryRun *q = A.run;
  const unsigned c = min(q->count[sel][0], (unsigned)A.n);
  const int k = max((int)(A.n * 0.95) - 1, 0), before = A.n - (int)c;
  if (t < 256) hist[0][t] = 0;
  cl.sync();  // every block has read the count
  if (rank == 0 && t == 0) q->count[sel][0] = 0;
  if (c == 0 || k < before) {  // (the same in every block)
    if (rank == 0 && t == 0) q->upd[sel] = 0;
    return;
  }
  const unsigned share = (c + kInjCluster - 1) / kInjCluster, lo = min(c, rank * share),
                 cnt = min(c, lo + share) - lo;
  const R *cand = A.cand + (long long)sel * A.n + lo;
  K *keys = reinterpret_cast<K *>(sm);
  const bool held = share * sizeof(K) <= (size_t)kInjSelectSmem;
  if (held)  // (a thread reads back its own entries only)
    for (unsigned j = t; j < cnt; j += kInjThreads) keys[j] = fkey(cand[j]);
  unsigned krem = (unsigned)(k - before);
  K prefix = 0;
  for (int b = KB - 8, p = 0; b >= 0; b -= 8, p ^= 1) {
    // the same trip count for every lane of a warp (for __match_any_sync)
    for (unsigned j0 = 0; j0 < cnt; j0 += kInjThreads) {
      const unsigned j = j0 + t;
      unsigned bin = 256u;
      if (j < cnt) {
        const K key = held ? keys[j] : fkey(cand[j]);
        if (b == KB - 8 || ((key ^ prefix) >> (b + 8)) == 0) bin = (unsigned)(key >> b) & 0xffu;
      }
      if (__all_sync(0xffffffffu, bin == 256u)) continue;
      const unsigned peers = __match_any_sync(0xffffffffu, bin);
      if (bin < 256u && lane == __ffs(peers) - 1) atomicAdd(&hist[p][bin], __popc(peers));
    }
    cl.sync();
    if (t < 256) {
      unsigned x = 0;
#pragma unroll
      for (int r = 0; r < kInjCluster; ++r) x += *cl.map_shared_rank(&hist[p][t], r);
      total[t] = x;
      hist[p ^ 1][t] = 0;
    }
    __syncthreads();
    if (t < 32) {  // eight bins per lane: the bin that holds the remaining rank
      unsigned h[8], sum = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        h[i] = total[8 * lane + i];
        sum += h[i];
      }
      unsigned x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      unsigned at = x - sum;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (krem >= at && krem < at + h[i]) {
          s_digit = 8 * lane + i;
          s_below = at;
        }
        at += h[i];
      }
    }
    __syncthreads();
    prefix |= (K)s_digit << b;
    krem -= s_below;
    __syncthreads();  // (s_digit, s_below before the next pass writes them)
  }
  cl.sync();  // no block leaves while another reads its histogram
  if (rank != 0 || t != 0) return;
  const double v = double(fkey_inv(prefix));
  q->upd[sel] = 1;
  q->v[sel] = q->run[sel] = v;
  q->vf[sel] = q->runf[sel] = float(v);
  const int count = (int)(c - ((unsigned)(k - before) - krem));  // candidates not below it
  InjuryState *s = A.state;
  if (sel == 0) {
    s->mps95 = v;
    s->mps95_time = time;
    s->mps95_count = count;
  } else {
    s->mpsxsr95 = v;
    s->mpsxsr95_time = time;
    s->mpsxsr95_count = count;
  }
}

// The step's extremes from the per-patch partials into the running state: a
// strictly better value takes the element and the time (the reference's
// ordered loop with strict comparisons).  Values are compared as
// order-preserving integers (FP64 compares issue once in 16 cycles).
template <class R>
__device__ __forceinline__ void injury_extremes(const InjuryArgs<R> &A, double time) {
  uint64_t key[4] = {0, 0, 0, 0};
  int jj[4] = {0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff}, cc[4] = {-1, -1, -1, -1};
  auto take = [&](int k, uint64_t x, int j, int c) {
    if (x > key[k] || (x == key[k] && j < jj[k])) {
      key[k] = x;
      jj[k] = j;
      cc[k] = c;
    }
  };
  for (int b = threadIdx.x; b < A.npart; b += kInjThreads) {
    const InjuryPart p = A.part[b];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint64_t x = fkey(p.v[k]);  // (never a NaN: injury_take)
      take(k, k == 1 ? ~x : x, p.j[k], p.c[k]);
    }
  }
  constexpr int NW = kInjThreads / 32;
  __shared__ uint64_t sk[4][NW];
  __shared__ int sj[4][NW], sc[4][NW];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto warp_best = [&]() {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint64_t x = __shfl_xor_sync(0xffffffffu, key[k], o);
        const int j = __shfl_xor_sync(0xffffffffu, jj[k], o);
        const int c = __shfl_xor_sync(0xffffffffu, cc[k], o);
        take(k, x, j, c);
      }
  };
  warp_best();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sk[k][w] = key[k];
      sj[k][w] = jj[k];
      sc[k][w] = cc[k];
    }
  }
  __syncthreads();
  if (w != 0) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    key[k] = sk[k][lane % NW];  // (twice is once for a maximum)
    jj[k] = sj[k][lane % NW];
    cc[k] = sc[k][lane % NW];
  }
  warp_best();
  if (lane != 0) return;
  InjuryState *s = A.state;
  double *val[4] = {&s->max_strain, &s->min_strain, &s->max_shear, &s->max_psxsr};
  double *tim[4] = {&s->max_strain_time, &s->min_strain_time, &s->max_shear_time,
                    &s->max_psxsr_time};
  int *el[4] = {&s->max_strain_elem, &s->min_strain_elem, &s->max_shear_elem, &s->max_psxsr_elem};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (cc[k] < 0) continue;
    const double v = fkey_inv(k == 1 ? ~key[k] : key[k]);
    const bool upd = (k == 1) ? (*val[k] > v) : (*val[k] < v);
    if (upd) {
      *val[k] = v;
      *el[k] = A.eref[cc[k]];
      *tim[k] = time;
    }
  }
  ++s->steps;
}

// The end of a step's criteria: clusters 0 and 1 the two percentiles, the
// first block of cluster 2 the extremes.
template <class R>
__global__ void __cluster_dims__(kInjCluster, 1, 1) __launch_bounds__(kInjThreads)
    k_injury_select(const InjuryArgs<R> A) {
  extern __shared__ __align__(16) unsigned char inj_sm[];
  const Clock ck = A.clock[A.parity];
  if (ck.done) return;
  const double time = ck.time + ck.dt;
  const int job = blockIdx.x / kInjCluster;
  if (job < 2)
    injury_select<R>(A, job, time, inj_sm);
  else if (blockIdx.x % kInjCluster == 0)
    injury_extremes<R>(A, time);
}

}  // namespace ftgpu
