// Row-wise norms either side of the GDPA forward, for the fused pipeline
//
//   ln_q = LayerNorm(Q) over all heads of a token      -> gdpa_layernorm_rows_kernel
//   x    = GDPA(ln_q, K, V) + ln_q                      (residual add and the per-row sum of x^2 are fused
//                                                        into the epilogue of gdpa_fwd_kernel)
//   out  = x * rsqrt(mean(x^2) + eps) * w (+ residual)  -> gdpa_rmsnorm_rows_kernel
//
// which is what the reference's GDPA-plus-norm kernel computes in one launch with a cluster of one CTA per
// head (gdpa_megakernel/src/tlx_gdpa_megakernel.py:359-405 RMS norm, :412-500 layer norm, :1076-1135
// epilogue order; checked by gdpa_megakernel/tests/test_tlx_gdpa_megakernel.py:50-145).  Both kernels are
// HBM-bound streaming passes: one warp per token row of N = heads * head_dim bf16 values, 16-byte loads,
// fp32 statistics, the row kept in registers between the statistics and the write when N <= 2048.  The backward
// of both norms (gdpa_norm_rows_bwd_kernel) holds a row in the registers of one to eight warps of a persistent grid.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "gdpa_launch.h"

namespace gdpa {

namespace {

constexpr int kNormThreads = 256;         // 8 rows per block

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f[2 * j] = __uint_as_float(w[j] << 16);
    f[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
  }
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}

__device__ __forceinline__ void load8(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// y = (x - mean) * rstd * weight + bias per row; mean and the (biased) variance over the N values of the row,
// variance from the centred values like torch.nn.functional.layer_norm.  A lane keeps up to kCachedChunks
// 16-byte chunks of the row in registers between the passes (rows of up to 256 * kCachedChunks values; the
// instantiation is chosen by the row length, fewer registers giving more rows in flight); longer rows are
// read again.
template <int kCachedChunks>
__global__ void __launch_bounds__(kNormThreads) gdpa_layernorm_rows_kernel(const NormArgs a) {
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * (kNormThreads / 32) + (threadIdx.x >> 5);
  if (row >= a.rows) return;
  const int chunks = a.n / 8;
  const uint4* src = reinterpret_cast<const uint4*>(a.x + row * a.n);
  uint4* dst = reinterpret_cast<uint4*>(a.out + row * a.n);
  const bool cached = chunks <= 32 * kCachedChunks;
  uint4 keep[kCachedChunks];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kCachedChunks; ++i) {
    const int c = lane + 32 * i;
    keep[i] = make_uint4(0, 0, 0, 0);
    if (c < chunks) {
      keep[i] = src[c];
      float f[8];
      unpack8(keep[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += f[j];
    }
  }
  for (int c = lane + 32 * kCachedChunks; c < chunks; c += 32) {
    float f[8];
    unpack8(src[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += f[j];
  }
  const float mean = warp_sum(sum) / static_cast<float>(a.n);
  float var = 0.f;
#pragma unroll
  for (int i = 0; i < kCachedChunks; ++i) {
    if (lane + 32 * i < chunks) {
      float f[8];
      unpack8(keep[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) var = fmaf(f[j] - mean, f[j] - mean, var);
    }
  }
  for (int c = lane + 32 * kCachedChunks; c < chunks; c += 32) {
    float f[8];
    unpack8(src[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) var = fmaf(f[j] - mean, f[j] - mean, var);
  }
  const float rstd = rsqrtf(warp_sum(var) / static_cast<float>(a.n) + a.eps);
  if (a.row_mean != nullptr && lane == 0) {
    a.row_mean[row] = mean;
    a.row_rstd[row] = rstd;
  }
  for (int c = lane; c < chunks; c += 32) {
    float f[8];
    const int i = c >> 5;
    uint4 v;
    if (cached) {
      // select from the register copy without dynamic indexing
      v = keep[0];
#pragma unroll
      for (int k = 1; k < kCachedChunks; ++k)
        if (i == k) v = keep[k];
    } else {
      v = src[c];
    }
    unpack8(v, f);
    float w[8], b[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      w[j] = 1.f;
      b[j] = 0.f;
    }
    if (a.weight != nullptr) load8(a.weight + 8 * c, w);
    if (a.bias != nullptr) load8(a.bias + 8 * c, b);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = fmaf((f[j] - mean) * rstd, w[j], b[j]);
    dst[c] = pack8(f);
  }
}

// out = x * rsqrt(sumsq / N + eps) * weight (+ residual).  `row_sumsq` holds the per-row sum of squares when
// the producer of x accumulated it (the forward kernel's fused epilogue); when it is null the kernel sums the
// squares of the bf16 values of x itself.
__global__ void __launch_bounds__(kNormThreads) gdpa_rmsnorm_rows_kernel(const NormArgs a) {
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * (kNormThreads / 32) + (threadIdx.x >> 5);
  if (row >= a.rows) return;
  const int chunks = a.n / 8;
  const uint4* src = reinterpret_cast<const uint4*>(a.x + row * a.n);
  uint4* dst = reinterpret_cast<uint4*>(a.out + row * a.n);
  const uint4* res = a.residual != nullptr ? reinterpret_cast<const uint4*>(a.residual + row * a.n) : nullptr;
  float ssq;
  if (a.row_sumsq != nullptr) {
    ssq = a.row_sumsq[row];
  } else {
    float s = 0.f;
    for (int c = lane; c < chunks; c += 32) {
      float f[8];
      unpack8(src[c], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) s = fmaf(f[j], f[j], s);
    }
    ssq = warp_sum(s);
  }
  const float rrms = rsqrtf(ssq / static_cast<float>(a.n) + a.eps);
  if (a.row_rstd != nullptr && lane == 0) a.row_rstd[row] = rrms;
  for (int c = lane; c < chunks; c += 32) {
    float f[8], w[8], r[8];
    unpack8(src[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      w[j] = 1.f;
      r[j] = 0.f;
    }
    if (a.weight != nullptr) load8(a.weight + 8 * c, w);
    if (res != nullptr) unpack8(res[c], r);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = fmaf(f[j] * rrms, w[j], r[j]);
    dst[c] = pack8(f);
  }
}

// ------------------------------------------------------------------------------------------------------------
// Backward of the two row norms.
//
// RMS norm  y = x r w,  r = rsqrt(mean(x^2) + eps)  (r saved by the forward):
//   g = dy w;  dx = r g - x r^3 mean(g x);  dw += dy x r.
// Layer norm  y = xh w + b  with xh = (x - mean) rstd (mean, rstd saved by the forward):
//   g = (dy + dy_add) w;  dx = rstd (g - mean(g) - xh mean(g xh));  dw += (dy + dy_add) xh;  db += dy + dy_add.
// `dy_add` is an optional second incoming gradient of the same shape (the Q-residual branch of the pipeline).
//
// HBM-bound if nothing but the rows moves: 2 or 3 row reads and one write of 2 bytes per value.  A row is held in the
// registers of WPR warps, two 16-byte chunks of every input per lane, so each byte is read once; a lane owns the same
// columns in every row its group takes, so the weight and bias gradients (sums over rows) are plain register sums for
// the whole kernel, added up over the block's groups in shared memory once at the end and flushed with one global
// atomic per column and block.  Before, every value of every row was a shared-memory atomic and the row was read twice:
// 543 us (RMS norm) and 957 us (layer norm) for 149 713 rows of 1024, now 188 and 257 us (floors at the copy rate 138 and
// 184 us); the whole forward and backward of that pipeline 8.52 -> 7.66 ms.
// Two chunks per lane keep the kernel under 80 (RMS norm) and 128 registers (layer norm), so three and two blocks of
// eight warps are resident and 48 KB of loads are in flight per SM.
constexpr int kNormBwdMaxN = 4096;  // 8 warps x 32 lanes x 2 chunks x 8 values; the gradients of w and b end there too

template <int MODE>
constexpr int kNormBwdResident = MODE == 1 ? 2 : 3;  // blocks per SM without spilled registers

template <int MODE, int WPR>  // MODE 0 = RMS norm, 1 = layer norm; WPR = warps per row (1, 2, 4, 8)
__global__ void __launch_bounds__(kNormThreads, kNormBwdResident<MODE>) gdpa_norm_rows_bwd_kernel(const NormBwdArgs a) {
  constexpr int kGroups = kNormThreads / 32 / WPR;  // rows a block works on at a time
  constexpr int kStride = 32 * WPR;                 // lanes of a group
  __shared__ float s_part[2][kNormThreads / 32][2];     // row sums of the warps of a group, by parity of the round
  __shared__ float s_acc[kGroups > 1 ? kGroups : 1][kStride][17];  // end of the kernel: one column sum set per group
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int group = warp / WPR;
  const int gl = threadIdx.x % kStride;  // lane within the group: chunks gl and gl + kStride of every row
  const int chunks = a.n / 8;
  const bool has[2] = {gl < chunks, gl + kStride < chunks};
  const float inv_n = 1.f / static_cast<float>(a.n);
  float dw[2][8], db[MODE == 1 ? 2 : 1][8];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dw[i][j] = 0.f;
      if (MODE == 1) db[i][j] = 0.f;
    }
  uint32_t round = 0;
  for (long long row0 = static_cast<long long>(blockIdx.x) * kGroups; row0 < a.rows;
       row0 += static_cast<long long>(gridDim.x) * kGroups, ++round) {
    const long long row = row0 + group;
    const bool live = row < a.rows;  // the same for every thread of a group
    uint4 g4[2], x4[2], e4[2];
    float rstd = 0.f, mean = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      g4[i] = x4[i] = e4[i] = make_uint4(0, 0, 0, 0);
      if (live && has[i]) {
        const long long at = row * chunks + gl + i * kStride;
        g4[i] = reinterpret_cast<const uint4*>(a.dy)[at];
        if (a.dy_add != nullptr) e4[i] = reinterpret_cast<const uint4*>(a.dy_add)[at];
        x4[i] = reinterpret_cast<const uint4*>(a.x)[at];
      }
    }
    if (live) {
      rstd = a.row_rstd[row];
      if (MODE == 1) mean = a.row_mean[row];
    }
    float g[2][8];  // the incoming gradient
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float e[8], x[8], w[8];
      unpack8(g4[i], g[i]);
      unpack8(e4[i], e);
      unpack8(x4[i], x);
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = 1.f;
      if (a.weight != nullptr && has[i]) load8(a.weight + 8 * (gl + i * kStride), w);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        g[i][j] += e[j];
        const float gw = g[i][j] * w[j];
        const float xh = MODE == 1 ? (x[j] - mean) * rstd : x[j];
        if (MODE == 1) s1 += gw;
        s2 = fmaf(gw, xh, s2);
        if (MODE == 1) {
          dw[i][j] = fmaf(g[i][j], xh, dw[i][j]);
          db[i][j] += g[i][j];
        } else {
          dw[i][j] = fmaf(g[i][j] * rstd, x[j], dw[i][j]);
        }
      }
    }
    if (MODE == 1) s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if constexpr (WPR > 1) {
      // two buffers: a warp that runs ahead into the next round writes the other one, and cannot run two rounds ahead
      // of a warp that has not passed this round's barrier
      float(*part)[2] = s_part[round & 1u];
      if (lane == 0) {
        part[warp][0] = s1;
        part[warp][1] = s2;
      }
      __syncthreads();
      s1 = s2 = 0.f;
#pragma unroll
      for (int k = 0; k < WPR; ++k) {
        s1 += part[group * WPR + k][0];
        s2 += part[group * WPR + k][1];
      }
    }
    s1 *= inv_n;
    s2 *= inv_n;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (live && has[i]) {
        float x[8], w[8], o[8];
        unpack8(x4[i], x);
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = 1.f;
        if (a.weight != nullptr) load8(a.weight + 8 * (gl + i * kStride), w);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float gw = g[i][j] * w[j];
          if (MODE == 0) o[j] = rstd * (gw - x[j] * rstd * rstd * s2);
          else o[j] = rstd * (gw - s1 - (x[j] - mean) * rstd * s2);
        }
        reinterpret_cast<uint4*>(a.dx)[row * chunks + gl + i * kStride] = pack8(o);
      }
    }
  }
  // column sums: over the groups of the block, then one atomic per column
#pragma unroll
  for (int t = 0; t < (MODE == 1 ? 2 : 1); ++t) {
    float* const out = t == 0 ? a.dweight : a.dbias;
    if (out == nullptr) continue;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) s_acc[group][gl][8 * i + j] = t == 0 ? dw[i][j] : db[MODE == 1 ? i : 0][j];
    __syncthreads();
    for (int c = threadIdx.x; c < a.n; c += kNormThreads) {
      const int chunk = c >> 3, i = chunk / kStride;
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < kGroups; ++k) v += s_acc[k][chunk - i * kStride][8 * i + (c & 7)];
      atomicAdd(out + c, v);
    }
  }
}

// dx = dy + dy_add (no norm): a stream of 16-byte chunks.
__global__ void __launch_bounds__(kNormThreads) gdpa_sum_rows_kernel(const NormBwdArgs a) {
  const long long n = a.rows * (a.n / 8), stride = static_cast<long long>(gridDim.x) * kNormThreads;
  for (long long c = static_cast<long long>(blockIdx.x) * kNormThreads + threadIdx.x; c < n; c += stride) {
    float f[8], g[8];
    unpack8(reinterpret_cast<const uint4*>(a.dy)[c], f);
    unpack8(reinterpret_cast<const uint4*>(a.dy_add)[c], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] += g[j];
    reinterpret_cast<uint4*>(a.dx)[c] = pack8(f);
  }
}

// The rows' gradients alone (no column sums, rows of any length): one warp per row, which reads the row twice, the second
// time from L1 / L2.  HBM-bound like the kernel above, but with 60 (RMS norm) and 48 registers four and five blocks are
// resident, so more rows are in flight, and a row need not fill the registers of whole warps.
template <int MODE>
__global__ void __launch_bounds__(kNormThreads) gdpa_norm_rows_bwd_wide_kernel(const NormBwdArgs a) {
  const int lane = threadIdx.x & 31;
  const int chunks = a.n / 8;
  const long long warps = static_cast<long long>(gridDim.x) * (kNormThreads / 32);
  const float inv_n = 1.f / static_cast<float>(a.n);
  for (long long row = static_cast<long long>(blockIdx.x) * (kNormThreads / 32) + (threadIdx.x >> 5); row < a.rows; row += warps) {
    const uint4* dy = reinterpret_cast<const uint4*>(a.dy + row * a.n);
    const uint4* dy2 = a.dy_add != nullptr ? reinterpret_cast<const uint4*>(a.dy_add + row * a.n) : nullptr;
    const uint4* x = reinterpret_cast<const uint4*>(a.x + row * a.n);
    uint4* dx = reinterpret_cast<uint4*>(a.dx + row * a.n);
    const float rstd = a.row_rstd[row];
    const float mean = MODE == 1 ? a.row_mean[row] : 0.f;
    // pass 1: the row sums
    float s1 = 0.f, s2 = 0.f;
    for (int c = lane; c < chunks; c += 32) {
      float g[8], xv[8], w[8];
      unpack8(dy[c], g);
      if (dy2 != nullptr) {
        float t[8];
        unpack8(dy2[c], t);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] += t[j];
      }
      unpack8(x[c], xv);
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = 1.f;
      if (a.weight != nullptr) load8(a.weight + 8 * c, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float gw = g[j] * w[j];
        const float xh = MODE == 1 ? (xv[j] - mean) * rstd : xv[j];
        s1 += gw;
        s2 = fmaf(gw, xh, s2);
      }
    }
    s1 = warp_sum(s1) * inv_n;
    s2 = warp_sum(s2) * inv_n;
    // pass 2: dx
    for (int c = lane; c < chunks; c += 32) {
      float g[8], xv[8], w[8], o[8];
      unpack8(dy[c], g);
      if (dy2 != nullptr) {
        float t[8];
        unpack8(dy2[c], t);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] += t[j];
      }
      unpack8(x[c], xv);
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = 1.f;
      if (a.weight != nullptr) load8(a.weight + 8 * c, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float gw = g[j] * w[j];
        if (MODE == 0) o[j] = rstd * (gw - xv[j] * rstd * rstd * s2);
        else o[j] = rstd * (gw - s1 - (xv[j] - mean) * rstd * s2);
      }
      dx[c] = pack8(o);
    }
  }
}

template <int MODE>
void launch_norm_bwd_mode(const NormBwdArgs& a, cudaStream_t stream) {
  // warps per row: the fewest that hold the row, 512 values each
  const int wpr = a.n <= 512 ? 1 : a.n <= 1024 ? 2 : a.n <= 2048 ? 4 : 8;
  // Without column sums the register kernel is the faster one only where the row fills its lanes: by three quarters where no
  // barrier is waited for (one warp) or the second reading would come from L2 (eight), and then for both norms; in between
  // by more than 7/8 and for the RMS norm.  2^27 values, register kernel and the other one: RMS norm 64 values a row 825 and
  // 695 us, 520: 284 and 221, 512: 168 and 195, 1024: 180 and 188, 3072: 205 and 254; layer norm 64: 1153 and 711, 1024: 227
  // and 185, 2056: 342 and 209, 3584: 239 and 275.
  const int held = 512 * wpr;
  const bool sums = a.dweight != nullptr || (MODE == 1 && a.dbias != nullptr);
  const bool filled = 4 * a.n >= 3 * held && (wpr == 1 || wpr == 8 || (MODE == 0 && 8 * a.n > 7 * held));
  if (a.n > kNormBwdMaxN || (!sums && !filled)) {
    // two rounds of the resident blocks; of the longer rows of the layer norm, which evict one another from L1, one per warp
    const long long most = MODE == 0 ? 148 * 8 : a.n <= 1536 ? 148 * 10 : 1 << 30;
    const long long blocks = (a.rows + kNormThreads / 32 - 1) / (kNormThreads / 32);
    gdpa_norm_rows_bwd_wide_kernel<MODE><<<static_cast<unsigned>(blocks < most ? blocks : most), kNormThreads, 0, stream>>>(a);
    return;
  }
  const int groups = kNormThreads / 32 / wpr;
  const long long most = 148 * kNormBwdResident<MODE>;  // every block flushes its column sums once
  const long long blocks = (a.rows + groups - 1) / groups;
  const unsigned grid = static_cast<unsigned>(blocks < most ? blocks : most);
  if (wpr == 1) gdpa_norm_rows_bwd_kernel<MODE, 1><<<grid, kNormThreads, 0, stream>>>(a);
  else if (wpr == 2) gdpa_norm_rows_bwd_kernel<MODE, 2><<<grid, kNormThreads, 0, stream>>>(a);
  else if (wpr == 4) gdpa_norm_rows_bwd_kernel<MODE, 4><<<grid, kNormThreads, 0, stream>>>(a);
  else gdpa_norm_rows_bwd_kernel<MODE, 8><<<grid, kNormThreads, 0, stream>>>(a);
}

}  // namespace

int launch_layernorm_rows(const NormArgs& a, cudaStream_t stream) {
  if (a.rows == 0) return 0;
  const long long blocks = (a.rows + kNormThreads / 32 - 1) / (kNormThreads / 32);
  const unsigned grid = static_cast<unsigned>(blocks);
  if (a.n <= 512) gdpa_layernorm_rows_kernel<2><<<grid, kNormThreads, 0, stream>>>(a);
  else if (a.n <= 1024) gdpa_layernorm_rows_kernel<4><<<grid, kNormThreads, 0, stream>>>(a);
  else gdpa_layernorm_rows_kernel<8><<<grid, kNormThreads, 0, stream>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : GDPA_ERR_LAUNCH_;
}

int launch_rmsnorm_rows(const NormArgs& a, cudaStream_t stream) {
  if (a.rows == 0) return 0;
  const long long blocks = (a.rows + kNormThreads / 32 - 1) / (kNormThreads / 32);
  gdpa_rmsnorm_rows_kernel<<<static_cast<unsigned>(blocks), kNormThreads, 0, stream>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : GDPA_ERR_LAUNCH_;
}

// mode: 0 = RMS norm, 1 = layer norm, 2 = plain sum of the two incoming gradients
int launch_norm_rows_bwd(const NormBwdArgs& a, int mode, cudaStream_t stream) {
  if (a.rows == 0) return 0;
  if (mode == 0) launch_norm_bwd_mode<0>(a, stream);
  else if (mode == 1) launch_norm_bwd_mode<1>(a, stream);
  else {
    const long long blocks = (a.rows * (a.n / 8) + kNormThreads - 1) / kNormThreads;
    gdpa_sum_rows_kernel<<<static_cast<unsigned>(blocks < 148 * 8 ? blocks : 148 * 8), kNormThreads, 0, stream>>>(a);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : GDPA_ERR_LAUNCH_;
}

}  // namespace gdpa
