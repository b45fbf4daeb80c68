// ft_train_tc.cuh -- one training step of the surrogate on the
// fifth-generation tensor cores: three launches per batch.  Included by
// ft_mlp.cu after its tcgen05 helpers.
//
//   k_train_rows   forward, loss and the backward data chain of 128 batch rows
//   k_train_dw     weight gradients of 256 batch rows, one layer per CTA
//   k_train_apply  the slices' sum, bias gradients, loss and Adam
//
// A batch of 8192 rows is 1.8 GFLOP, about a microsecond of the tensor cores:
// what bounds a step is its chain of layers and the launches.  One launch per
// GEMM (25 launches a batch, FP32 pre-activations through memory row by row,
// transposed operands gathered two bytes at a time) took 545 us a batch; here
// a CTA carries its rows through all layers and back on the chip, and the
// operands of the weight gradients leave it in the layout their MMAs read:
// 47 us a batch (k_train_rows 27 us on 64 CTAs, of which its seven dependent
// layers are the bound; 36 us with 256 threads; k_train_dw and k_train_apply
// 7 us each).
//
// Bitwise reproducible, and bit for bit the arithmetic of one GEMM per launch:
// every accumulator adds its K = 16 steps in ascending order, weight
// gradients are split over the batch in slices of 256 rows (one slice up to
// 512 rows) and the FP32 slices are added in order.
#pragma once

namespace trn {
constexpr int kThreads = 512;                // k_train_rows
constexpr int kDwThreads = 256;              // k_train_dw
// K-major core-matrix images without swizzle: element (r, k) of an image of K
// columns at (r / 8) * 16 K + (k / 8) * 128 + (r % 8) * 16 + (k % 8) * 2
constexpr uint32_t kImgH = 128 * 128 * 2, kImgX = 128 * 16 * 2;  // [128 x 128], [128 x 16]
constexpr uint32_t kW0 = 0;                  // [128 x 16]
constexpr uint32_t kW1 = kW0 + kImgX;        // [128 x 128]
constexpr uint32_t kW2 = kW1 + kImgH;        // [128 x 128]
constexpr uint32_t kW3 = kW2 + kImgH;        // [16 x 128], rows 8..15 zero
constexpr uint32_t kW1T = kW3 + kImgX;       // the transposes, operands of the way back
constexpr uint32_t kW2T = kW1T + kImgH;
constexpr uint32_t kW3T = kW2T + kImgH;      // [128 x 16], columns 8..15 zero
constexpr uint32_t kX = kW3T + kImgX;        // rows' features, later dY: [128 x 16]
constexpr uint32_t kH = kX + kImgX;          // activations, later dZ: [128 x 128]
constexpr uint32_t kBias = kH + kImgH;       // b0 b1 b2 (128 each), b3 (8)
constexpr uint32_t kBar = kBias + 4 * (3 * 128 + 8);
constexpr uint32_t kSmemRows = kBar + 16 + 128;  // + alignment slack of the base
// accumulators: Z1, Z2, Z3 stay in tensor memory from the forward pass until
// the backward pass has used them; the fourth block is Y and then dH
constexpr uint32_t kWork = 384, kTmemCols = 512;
// transposed operand images of one 128-row tile in global memory (bytes):
// X^T [16 x 128], H1^T..H3^T and dZ1^T..dZ3^T [128 x 128], dY^T [8 x 128]
constexpr size_t kTileX = 0, kTileH = kImgX, kTileZ = kTileH + 3 * kImgH,
                 kTileY = kTileZ + 3 * kImgH, kTileBytes = kTileY + 8 * 128 * 2;
constexpr int kSlice = 256;                  // batch rows of one weight-gradient slice
constexpr uint32_t kDwA = 0, kDwB = 2 * kImgH, kDwBar = 4 * kImgH,
                   kSmemDw = kDwBar + 48 + 128;
constexpr int kDwPitch = 132;                // FP32 row pitch of the staged result
static_assert(128 * kDwPitch * 4 <= kDwBar, "staged result fits the operand images");
}  // namespace trn

// Batch rows of one weight-gradient slice and the slices of a batch
__host__ __device__ inline int train_slice_rows(long long n) {
  return n > 512 ? trn::kSlice : 512;
}

// Four 8 x 8 core matrices read transposed; a store of register i by the
// whole warp (32 consecutive words) is the transposed core matrix i.
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&v)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(saddr)
               : "memory");
}

// Transpose of the first `ncol` columns of a [128 x K] image into dst
// (word core (k / 8, r / 8) * 32 + lane), four cores per warp and step.
template <int K>
__device__ __forceinline__ void trn_transpose(uint32_t img, uint32_t *dst, int ncol) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = warp; i < 4 * (ncol / 8); i += trn::kThreads / 32) {
    const int ci = i >> 2, r4 = 4 * (i & 3);  // column group, first of four row groups
    uint32_t v[4];
    ldmatrix_x4_trans(v, img + (uint32_t)((r4 + (lane >> 3)) * 16 * K + ci * 128 + (lane & 7) * 16));
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[(ci * 16 + r4 + j) * 32 + lane] = v[j];
  }
}

// A row-major BF16 matrix [rows x K] into a [rows_pad x Ki] image, zero outside
__device__ __forceinline__ void trn_stage(unsigned char *img, const bf16 *src, int rows, int K,
                                          int rows_pad, int Ki) {
  for (int d = threadIdx.x; d < rows_pad * Ki / 8; d += trn::kThreads) {
    const int r = d / (Ki / 8), q = d - r * (Ki / 8);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (r < rows && 8 * q < K) v = *reinterpret_cast<const uint4 *>(src + r * K + 8 * q);
    *reinterpret_cast<uint4 *>(img + (r >> 3) * 16 * Ki + q * 128 + (r & 7) * 16) = v;
  }
}

// D = A B^T over K / 16 steps, committed to the barrier (one thread)
template <int K>
__device__ __forceinline__ void trn_issue(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc,
                                          uint32_t bar) {
  tc_fence_after();
#pragma unroll
  for (int kk = 0; kk < K / 16; ++kk)
    umma_bf16(tmem_d, umma_sdesc(a + 256 * kk, 128, 16 * K), umma_sdesc(b + 256 * kk, 128, 16 * K),
              idesc, kk > 0 ? 1u : 0u);
  umma_commit(bar);
}

// Forward (and, BWD, loss and backward data) of 128-row tiles.  512 threads:
// warp w reads TMEM lanes 32 (w % 4) .. + 31 (one batch row per thread) and
// columns 32 (w / 4) .. + 31.  Per layer: the operand image is complete ->
// one thread issues the MMAs -> meanwhile all warps write the image's
// transpose to memory for the weight gradients -> the accumulator comes back
// through the activation (or its derivative) as the next operand image.
template <bool BWD>
__global__ void __launch_bounds__(trn::kThreads, 1)
    k_train_rows(const bf16 *__restrict__ X, const float *__restrict__ T, long long n,
                 const bf16 *__restrict__ Wg, const float *__restrict__ P, float *__restrict__ Y,
                 float *__restrict__ rowloss, unsigned char *__restrict__ tiles, int *err) {
  extern __shared__ __align__(128) unsigned char trn_raw[];
  unsigned char *sm = trn_raw + ((128 - (smem_u32(trn_raw) & 127)) & 127);
  const uint32_t sb = smem_u32(sm);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const uint32_t bar = sb + trn::kBar;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + trn::kBar + 8);
  volatile int *abort = reinterpret_cast<volatile int *>(sm + trn::kBar + 12);
  float *bias = reinterpret_cast<float *>(sm + trn::kBias);
  trn_stage(sm + trn::kW0, Wg + kOffW0, kMlpHid, kMlpIn, 128, 16);
  trn_stage(sm + trn::kW1, Wg + kOffW1, kMlpHid, kMlpHid, 128, 128);
  trn_stage(sm + trn::kW2, Wg + kOffW2, kMlpHid, kMlpHid, 128, 128);
  trn_stage(sm + trn::kW3, Wg + kOffW3, kMlpOut, kMlpHid, 16, 128);
  if (BWD)  // W3^T: row k holds the eight outputs' weights of hidden unit k
    for (int k = t; k < kMlpHid; k += trn::kThreads) {
      uint4 v;
      bf16 *e = reinterpret_cast<bf16 *>(&v);
#pragma unroll
      for (int j = 0; j < 8; ++j) e[j] = Wg[kOffW3 + j * kMlpHid + k];
      unsigned char *d = sm + trn::kW3T + (k >> 3) * 256 + (k & 7) * 16;
      *reinterpret_cast<uint4 *>(d) = v;
      *reinterpret_cast<uint4 *>(d + 128) = make_uint4(0u, 0u, 0u, 0u);
    }
  if (t < kMlpHid) {
    bias[t] = P[kOffB0 + t];
    bias[128 + t] = P[kOffB1 + t];
    bias[256 + t] = P[kOffB2 + t];
    if (t < kMlpOut) bias[384 + t] = P[kOffB3 + t];
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(trn::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (BWD) {
    trn_transpose<128>(sb + trn::kW1, reinterpret_cast<uint32_t *>(sm + trn::kW1T), 128);
    trn_transpose<128>(sb + trn::kW2, reinterpret_cast<uint32_t *>(sm + trn::kW2T), 128);
  }
  const uint32_t tmem = *tmem_slot;
  const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);  // this warp's lanes
  const int r = 32 * (warp & 3) + lane, part = warp >> 2;
  constexpr uint32_t id128 = umma_idesc_bf16(128, 128), id16 = umma_idesc_bf16(128, 16);
  unsigned char *hrow = sm + trn::kH + (r >> 3) * 2048 + (r & 7) * 16;
  unsigned char *xrow = sm + trn::kX + (r >> 3) * 256 + (r & 7) * 16;
  const long long ntile = (n + 127) / 128;
  uint32_t phase = 0;
  bool ok = true;
  // the operand image is written: make it visible to the tensor core
  auto publish = [&]() {
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
  };
  // the MMAs of this layer are done, and with them (and every warp's
  // transpose) the operand image is free; false: a wait gave up
  auto arrived = [&]() {
    const bool got = mbar_wait(bar, phase, abort);
    phase ^= 1u;
    tc_fence_after();
    __syncthreads();
    ok = ok && got && !*abort;
    return ok;
  };
  for (long long tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
    const long long row = tile * 128 + r;
    unsigned char *to = BWD ? tiles + tile * trn::kTileBytes : nullptr;
    if (part == 0) {
      uint4 xa = make_uint4(0u, 0u, 0u, 0u), xb = xa;
      if (row < n) {
        const uint4 *src = reinterpret_cast<const uint4 *>(X + row * kMlpIn);
        xa = src[0];
        xb = src[1];
      }
      *reinterpret_cast<uint4 *>(xrow) = xa;
      *reinterpret_cast<uint4 *>(xrow + 128) = xb;
    }
    publish();
    if (t == 0) trn_issue<16>(tmem, sb + trn::kX, sb + trn::kW0, id128, bar);
    if (BWD) trn_transpose<16>(sb + trn::kX, reinterpret_cast<uint32_t *>(to + trn::kTileX), 16);
    // hidden layers: activation of layer l, then its product with the next weights
#pragma unroll 1
    for (int l = 0; l < 3; ++l) {
      if (!arrived()) break;
      {
        const int c0 = 32 * part;
        float v[32];
        tmem_ld32(tl + 128u * l + c0, v);
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
          pk[j] = silu_bf16x2(v[2 * j] + bias[128 * l + c0 + 2 * j],
                              v[2 * j + 1] + bias[128 * l + c0 + 2 * j + 1]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4 *>(hrow + (c0 / 8 + i) * 128) =
              make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
      }
      publish();
      if (t == 0) {
        if (l < 2)
          trn_issue<128>(tmem + 128u * (l + 1), sb + trn::kH, sb + (l ? trn::kW2 : trn::kW1),
                         id128, bar);
        else
          trn_issue<128>(tmem + trn::kWork, sb + trn::kH, sb + trn::kW3, id16, bar);
      }
      if (BWD)
        trn_transpose<128>(sb + trn::kH,
                           reinterpret_cast<uint32_t *>(to + trn::kTileH + l * trn::kImgH), 128);
    }
    if (!ok || !arrived()) break;
    {  // outputs, loss of the row and dY = 2 (Y - T) / (used outputs * batch)
      float y[16];
      tmem_ld16(tl + trn::kWork, y);
      if (part == 0) {
        uint32_t dp[4] = {0u, 0u, 0u, 0u};
        if (row < n) {
#pragma unroll
          for (int k = 0; k < kMlpOut; ++k) y[k] += bias[384 + k];
          float4 *yd = reinterpret_cast<float4 *>(Y + row * kMlpOut);
          yd[0] = make_float4(y[0], y[1], y[2], y[3]);
          yd[1] = make_float4(y[4], y[5], y[6], y[7]);
          if (BWD) {
            const float4 *td = reinterpret_cast<const float4 *>(T + row * kMlpOut);
            const float4 ta = td[0], tb = td[1];
            const float tt[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
            const float sc = 2.f / (float(kMlpUsedOut) * float(n));
            float l = 0.f;
            bf16 dy[8];
#pragma unroll
            for (int k = 0; k < kMlpOut; ++k) {
              const float d = k < kMlpUsedOut ? y[k] - tt[k] : 0.f;
              l += d * d;
              dy[k] = __float2bfloat16_rn(sc * d);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) dp[k] = pack2(dy[2 * k], dy[2 * k + 1]);
            rowloss[row] = l;
          }
        }
        if (BWD) {
          *reinterpret_cast<uint4 *>(xrow) = make_uint4(dp[0], dp[1], dp[2], dp[3]);
          *reinterpret_cast<uint4 *>(xrow + 128) = make_uint4(0u, 0u, 0u, 0u);
        }
      }
    }
    publish();
    if (!BWD) continue;
    if (t == 0) trn_issue<16>(tmem + trn::kWork, sb + trn::kX, sb + trn::kW3T, id128, bar);
    trn_transpose<16>(sb + trn::kX, reinterpret_cast<uint32_t *>(to + trn::kTileY), 8);
    // dZ_l = (dZ_{l+1} W_{l+1}) silu'(Z_l), l = 3, 2, 1
#pragma unroll 1
    for (int l = 2; l >= 0; --l) {
      if (!arrived()) break;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        const int c0 = 32 * part + 16 * c;
        float v[16], z[16];
        tmem_ld16(tl + trn::kWork + c0, v);
        tmem_ld16(tl + 128u * l + c0, z);
        uint32_t pk[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          pk[j] = pack2(
              __float2bfloat16_rn(v[2 * j] * dsilu(z[2 * j] + bias[128 * l + c0 + 2 * j])),
              __float2bfloat16_rn(v[2 * j + 1] * dsilu(z[2 * j + 1] + bias[128 * l + c0 + 2 * j + 1])));
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<uint4 *>(hrow + (c0 / 8 + i) * 128) =
              make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
      }
      publish();
      if (t == 0 && l > 0)
        trn_issue<128>(tmem + trn::kWork, sb + trn::kH, sb + (l == 2 ? trn::kW2T : trn::kW1T),
                       id128, bar);
      trn_transpose<128>(sb + trn::kH,
                         reinterpret_cast<uint32_t *>(to + trn::kTileZ + l * trn::kImgH), 128);
    }
    __syncthreads();  // the last transpose has read the image
  }
  if (!ok && t == 0) atomicOr(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(trn::kTmemCols)
                 : "memory");
}

// dW_l of one batch slice: dW = dZ^T H, both operands transposed images as
// k_train_rows left them, so a tile is two bulk copies and eight MMAs.
// blockIdx.y: layer 0..3 (operand rows dZ1, dZ2, dZ3, dY; columns X, H1, H2,
// H3).  The FP32 result is staged through shared memory for whole-row stores
// into part[slice][parameter].
__global__ void __launch_bounds__(trn::kDwThreads, 1)
    k_train_dw(const unsigned char *__restrict__ tiles, long long n, float *__restrict__ part,
               int *err) {
  extern __shared__ __align__(128) unsigned char trn_raw[];
  unsigned char *sm = trn_raw + ((128 - (smem_u32(trn_raw) & 127)) & 127);
  const uint32_t sb = smem_u32(sm);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, l = blockIdx.y;
  const uint32_t full = sb + trn::kDwBar, done = full + 16;  // two of each, by buffer
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + trn::kDwBar + 32);
  volatile int *abort = reinterpret_cast<volatile int *>(sm + trn::kDwBar + 36);
  const int rows = train_slice_rows(n);
  const long long first = (long long)blockIdx.x * rows / 128;
  const long long ntile = (n + 127) / 128;
  const int nt = (int)min((long long)(rows / 128), ntile - first);
  const size_t offA = l == 3 ? trn::kTileY : trn::kTileZ + l * (size_t)trn::kImgH;
  const size_t offB = l == 0 ? trn::kTileX : trn::kTileH + (l - 1) * (size_t)trn::kImgH;
  const uint32_t szA = l == 3 ? 8 * 128 * 2 : trn::kImgH, szB = l == 0 ? trn::kImgX : trn::kImgH;
  if (l == 3)  // dY^T has eight rows: the rest of the operand's 128 rows is zero
    for (uint32_t d = 16 * t; d < 2 * trn::kImgH; d += 16 * trn::kDwThreads)
      *reinterpret_cast<uint4 *>(sm + trn::kDwA + d) = make_uint4(0u, 0u, 0u, 0u);
  if (t == 0) {
    for (int b = 0; b < 4; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + 8 * b) : "memory");
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(128)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t idesc = umma_idesc_bf16(128, l == 0 ? 16 : 128);
  if (t == 0) {
    auto load = [&](int i) {
      const uint32_t b = i & 1, fb = full + 8 * b;
      const unsigned char *src = tiles + (first + i) * trn::kTileBytes;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(szA + szB)
                   : "memory");
      bulk_load(sb + trn::kDwA + b * trn::kImgH, src + offA, szA, fb);
      bulk_load(sb + trn::kDwB + b * trn::kImgH, src + offB, szB, fb);
    };
    int loaded = 0;
    for (; loaded < nt && loaded < 2; ++loaded) load(loaded);
    bool ok = true;
    for (int i = 0; i < nt && ok; ++i) {
      const uint32_t b = i & 1, ph = (i >> 1) & 1;
      ok = mbar_wait(full + 8 * b, ph, abort);
      if (!ok) break;
      const uint32_t a = sb + trn::kDwA + b * trn::kImgH, h = sb + trn::kDwB + b * trn::kImgH;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16(tmem, umma_sdesc(a + 256 * kk, 128, 2048), umma_sdesc(h + 256 * kk, 128, 2048),
                  idesc, (i > 0 || kk > 0) ? 1u : 0u);
      umma_commit(done + 8 * b);
      if (loaded < nt) {  // the buffer is free once its MMAs are done
        ok = mbar_wait(done + 8 * b, ph, abort);
        if (ok) load(loaded++);
      }
    }
    // the last commit covers every MMA before it
    if (ok) ok = mbar_wait(done + 8 * ((nt - 1) & 1), ((nt - 1) >> 1) & 1, abort);
    if (!ok) {
      atomicOr(err, 1);
      *abort = 1;
      // copies already issued (bounded): nothing may land after the block has left
      for (int i = max(0, loaded - 2); i < loaded; ++i)
        for (int w = 0; w < tc::kWaitLimit; ++w) {
          uint32_t got;
          asm volatile(
              "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
              "selp.u32 %0, 1, 0, p;\n\t}\n"
              : "=r"(got)
              : "r"(full + 8 * (i & 1)), "r"((uint32_t)((i >> 1) & 1))
              : "memory");
          if (got) break;
        }
    }
  }
  __syncthreads();
  tc_fence_after();
  if (!*abort) {
    const int r = 32 * (warp & 3) + lane, half = warp >> 2;
    const int N = l == 0 ? kMlpIn : kMlpHid, M = l == 3 ? kMlpOut : kMlpHid;
    float *st = reinterpret_cast<float *>(sm);
    const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    for (int c0 = 64 * half; c0 < min(N, 64 * half + 64); c0 += 16) {
      float v[16];
      tmem_ld16(tl + (uint32_t)c0, v);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4 *>(st + r * trn::kDwPitch + c0 + 4 * i) =
            make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
    __syncthreads();
    const int off = l == 0 ? kOffW0 : l == 1 ? kOffW1 : l == 2 ? kOffW2 : kOffW3;
    float *dst = part + (long long)blockIdx.x * kMlpParams + off;
    for (int i = t; i < M * N / 4; i += trn::kDwThreads) {
      const int row = 4 * i / N, c = 4 * i - row * N;
      *reinterpret_cast<float4 *>(dst + 4 * i) =
          *reinterpret_cast<const float4 *>(st + row * trn::kDwPitch + c);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128)
                 : "memory");
}

// The offset of weight parameter w (0 .. weights - 1) in the parameter vector
constexpr int kTrnWeights = kMlpHid * kMlpIn + 2 * kMlpHid * kMlpHid + kMlpOut * kMlpHid;
constexpr int kTrnBiases = 3 * kMlpHid + kMlpOut;
constexpr int kTrnApplyW = (kTrnWeights + 255) / 256;  // blocks of weights

struct AdamArgs {
  int on;  // 0: gradient only
  float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ void adam_update(int i, float g, float *P, float *Mo, float *V,
                                            bf16 *Wb, const AdamArgs &a) {
  const float m = a.b1 * Mo[i] + (1.f - a.b1) * g;
  const float v = a.b2 * V[i] + (1.f - a.b2) * g * g;
  Mo[i] = m;
  V[i] = v;
  const float p = P[i] - a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
  P[i] = p;
  Wb[i] = __float2bfloat16_rn(p);
}

// Blocks 0 .. kTrnApplyW - 1: a weight per thread, its slices in order (all
// slices' loads of a thread are independent, consecutive threads read
// consecutive words).  The next kTrnBiases blocks: a bias gradient each, the
// column sum of dZ as strided per-thread sums and a fixed tree.  The last
// block: the loss.  Then Adam on the parameter in hand.
__global__ void __launch_bounds__(256)
    k_train_apply(const unsigned char *__restrict__ tiles, const float *__restrict__ part,
                  const float *__restrict__ rowloss, long long n, int slices, float *P, float *G,
                  float *Mo, float *V, bf16 *Wb, float *loss, const AdamArgs a) {
  const int t = threadIdx.x;
  if (blockIdx.x < kTrnApplyW) {
    const int w = blockIdx.x * 256 + t;
    if (w >= kTrnWeights) return;
    constexpr int n0 = kMlpHid * kMlpIn, n1 = kMlpHid * kMlpHid;
    const int i = w < n0 ? kOffW0 + w
                         : w < n0 + n1 ? kOffW1 + w - n0
                                       : w < n0 + 2 * n1 ? kOffW2 + w - n0 - n1
                                                         : kOffW3 + w - n0 - 2 * n1;
    float s = 0.f;
#pragma unroll 16
    for (int k = 0; k < slices; ++k) s += part[(long long)k * kMlpParams + i];
    G[i] = s;
    if (a.on) adam_update(i, s, P, Mo, V, Wb, a);
    return;
  }
  __shared__ float red[256];
  const int b = blockIdx.x - kTrnApplyW;
  float s = 0.f;
  int i = -1;
  if (b < kTrnBiases) {
    const int l = b / kMlpHid, c = b - l * kMlpHid;
    i = (l == 0 ? kOffB0 : l == 1 ? kOffB1 : l == 2 ? kOffB2 : kOffB3) + c;
    const size_t off = l == 3 ? trn::kTileY : trn::kTileZ + l * (size_t)trn::kImgH;
    // element (c, r) of the transposed image of a tile, r = t % 128
    const int r = t & 127;
    const unsigned char *src = tiles + (t >> 7) * trn::kTileBytes + off +
                               ((c >> 3) * 16 + (r >> 3)) * 128 + (c & 7) * 16 + (r & 7) * 2;
#pragma unroll 16
    for (long long row = t; row < n; row += 256, src += 2 * trn::kTileBytes)
      s += __bfloat162float(*reinterpret_cast<const bf16 *>(src));
  } else {
#pragma unroll 8
    for (long long row = t; row < n; row += 256) s += rowloss[row];
  }
  red[t] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) red[t] += red[t + w];
    __syncthreads();
  }
  if (t != 0) return;
  if (i < 0) {
    *loss = red[0];
    return;
  }
  G[i] = red[0];
  if (a.on) adam_update(i, red[0], P, Mo, V, Wb, a);
}
