// HBM-bound row kernels: (add bias + residual +) LayerNorm, the same fused with
// the packed -> padded scatter, add-bias + GELU, and masked softmax.
//
// All of them use 16-byte global accesses and warp-shuffle reductions; one warp
// owns one row, so no shared memory or block barrier is needed.
//
// Reference counterparts (paths relative to the ByteTransformer root):
//   layernorm_rows_kernel<false>  add_bias_input_layernorm{,_v2}
//                                 (bytetransformer/include/layernorm.h:273-296, src/layernorm.cu:89-102)
//   layernorm_rows_kernel<true>   add_bias_input_layernorm_restore_output{,_v2}
//                                 (layernorm.h:334-373, layernorm.cu:126-148)
//   add_bias_gelu_kernel          add_bias_gelu (bytetransformer/src/gemm_bias_act.cu:32-47)
//   masked_softmax_kernel         softmax_kernel_warp_half2* (bytetransformer/include/softmax.h:25-297)
// Differences kept on purpose: the sums x + bias + residual are formed in fp32
// (the reference adds in fp16 first, layernorm.h:289-290); statistics are
// two-pass (mean, then centred variance) in fp32 as in the reference.
//
// Algorithmic bytes per row of H halves: LayerNorm reads x (+ residual) and
// writes out: 6*H bytes with residual, 4*H without; the restore variant writes
// every padded row (2*H bytes each, zeros for padding).
#include "common.cuh"
#include "kernels.h"
#include "../../include/bt_b200.h"

namespace bt {

namespace {

constexpr int kLnWarps = 4;
constexpr int kLnMaxVec = 4;  // register-resident rows up to 4*32*8 = 1024 halves
constexpr int kLnMaxSplit = 8;  // most fp32 partial sums a row may arrive in

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ void unpack8(const uint4& q, float (&f)[8]) {
  const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __half22float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 q;
  q.x = pack_half2(f[0], f[1]);
  q.y = pack_half2(f[2], f[3]);
  q.z = pack_half2(f[4], f[5]);
  q.w = pack_half2(f[6], f[7]);
  return q;
}

template <bool GB_FP32>
__device__ __forceinline__ void load_gb8(const void* p, int vec, float (&f)[8]) {
  if (GB_FP32) {
    const float4* fp = reinterpret_cast<const float4*>(p) + 2 * vec;
    const float4 a = __ldg(fp), b = __ldg(fp + 1);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  } else {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(p) + vec);
    unpack8(q, f);
  }
}

// RESTORE = false: rows [0, M) of x -> rows [0, M) of out.
// RESTORE = true : grid covers the B*S padded rows; row (b,i) reads packed row
//                  batch_idx[b]+i when i < len_b, else writes zeros.
template <bool RESTORE, bool GB_FP32, bool X_FP32, int NVEC>
__global__ void __launch_bounds__(kLnWarps * 32)
layernorm_rows_kernel(const void* __restrict__ x_v, const __half* __restrict__ bias,
                      const __half* __restrict__ residual, const void* __restrict__ gamma,
                      const void* __restrict__ beta, __half* __restrict__ out, const int* __restrict__ m_dev,
                      int m_rows, const int* __restrict__ batch_idx, int S, int hidden, float eps) {
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nvec = hidden / 8;
  {
    // gamma and beta are written by no kernel of the chain: ask for their lines while waiting
    const int gb_bytes = hidden * (GB_FP32 ? 4 : 2);
    const int off = static_cast<int>(threadIdx.x) * 128;
    if (off < gb_bytes) {
      prefetch_l1(reinterpret_cast<const uint8_t*>(gamma) + off);
      prefetch_l1(reinterpret_cast<const uint8_t*>(beta) + off);
    }
  }
  pdl_wait();
  // Rows are walked with a grid stride (the grid is capped at a few waves of the machine), so
  // a warp keeps streaming instead of paying a block launch per row.
  long long row_limit = m_rows;
  if (!RESTORE && m_dev != nullptr) {
    const int md = __ldg(m_dev);
    row_limit = md < m_rows ? md : m_rows;
  }
  // A warp's first row is read before the row count has arrived (it lies inside the allocation either way) and
  // dropped after the first reduction if it does not exist: in a call of a few rows the count's L2 round trip is a
  // tenth of the kernel.
  const long long first_row = static_cast<long long>(blockIdx.x) * kLnWarps + warp;
  for (long long row = first_row; row < (row == first_row ? m_rows : row_limit);
       row += static_cast<long long>(gridDim.x) * kLnWarps) {
  long long src_row = row;
  if (RESTORE) {
    const int b = static_cast<int>(row / S);
    const int i = static_cast<int>(row - static_cast<long long>(b) * S);
    const int off = __ldg(batch_idx + b);
    const int len = __ldg(batch_idx + b + 1) - off;
    if (i >= len) {
      uint4* o4 = reinterpret_cast<uint4*>(out + row * hidden);
      for (int v = lane; v < nvec; v += 32) o4[v] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    src_row = off + i;
  }

  const uint4* x4 = reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(x_v) + src_row * hidden);
  const float4* xf = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x_v) + src_row * hidden);
  const uint4* r4 = residual ? reinterpret_cast<const uint4*>(residual + src_row * hidden) : nullptr;
  const uint4* b4 = bias ? reinterpret_cast<const uint4*>(bias) : nullptr;

  float val[NVEC][8];
  float sum = 0.f;
#pragma unroll
  for (int it = 0; it < NVEC; ++it) {
    const int v = it * 32 + lane;
    if (v < nvec) {
      if (X_FP32) {
        const float4 a = __ldg(xf + 2 * v), b = __ldg(xf + 2 * v + 1);
        val[it][0] = a.x; val[it][1] = a.y; val[it][2] = a.z; val[it][3] = a.w;
        val[it][4] = b.x; val[it][5] = b.y; val[it][6] = b.z; val[it][7] = b.w;
      } else {
        unpack8(__ldg(x4 + v), val[it]);
      }
      if (r4) {
        float t[8];
        unpack8(__ldg(r4 + v), t);
#pragma unroll
        for (int k = 0; k < 8; ++k) val[it][k] += t[k];
      }
      if (b4) {
        float t[8];
        unpack8(__ldg(b4 + v), t);
#pragma unroll
        for (int k = 0; k < 8; ++k) val[it][k] += t[k];
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += val[it][k];
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) val[it][k] = 0.f;
    }
  }
  const float mean = warp_sum(sum) / static_cast<float>(hidden);
  if (!RESTORE && row >= row_limit) break;
  float sq = 0.f;
#pragma unroll
  for (int it = 0; it < NVEC; ++it) {
    if (it * 32 + lane < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = val[it][k] - mean;
        sq = fmaf(d, d, sq);
      }
    }
  }
  const float rstd = rsqrtf(warp_sum(sq) / static_cast<float>(hidden) + eps);

  uint4* o4 = reinterpret_cast<uint4*>(out + row * hidden);
#pragma unroll
  for (int it = 0; it < NVEC; ++it) {
    const int v = it * 32 + lane;
    if (v < nvec) {
      float g[8], bt_[8], o[8];
      load_gb8<GB_FP32>(gamma, v, g);
      load_gb8<GB_FP32>(beta, v, bt_);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = fmaf((val[it][k] - mean) * rstd, g[k], bt_[k]);
      o4[v] = pack8(o);
    }
  }
  }  // row loop
}

// The same for the fp32 sums that a GEMM left (no bias, no residual): a CTA holds one row, or ROWS of them, four columns
// per thread.  Such a kernel is a chain of latencies, not of bytes: a warp per row loads the up to eight partial sums of
// its columns in three rounds (48 16-byte loads per lane), here every thread has its loads in flight at once; gamma and
// beta are in registers before the dependency wait, and the code is a tenth of the length (a kernel that runs once per
// SM fetches every instruction from L2).  One row per CTA shortens the chain most; with more rows the statistics, which
// every warp forms for itself then, cost more issue slots than they save, and several rows share a CTA, a warp forming
// the statistics of each.  Measured, us per 12-layer forward, warp per row / one row / four rows per CTA (hidden 768, all
// rows valid): 88 rows 480 / 412 / -, 984 rows 745 / 708 / -, 1112 rows 687 / 689 / 662, 2008 rows 857 / 873 / 812,
// 4096 rows 1328 / 1405 / 1273, 8000 rows 2187 / 2460 / 2208.
template <bool RESTORE, bool GB_FP32, int SPLITS, int ROWS, int NVEC>
__global__ void __launch_bounds__(256)
layernorm_cta_kernel(const float* __restrict__ x, const void* __restrict__ gamma, const void* __restrict__ beta,
                     __half* __restrict__ out, const int* __restrict__ m_dev, int m_rows,
                     const int* __restrict__ batch_idx, int S, int hidden, float eps, LnSplit split) {
  // a row's sums, four columns per unit: even and odd units apart (by 64 bytes modulo the banks), so that a lane's eight
  // columns are two conflict-free reads
  __shared__ float4 vals[ROWS][2][NVEC * 32 + 4];
  __shared__ float2 stats[ROWS];  // mean, 1 / standard deviation
  pdl_launch_dependents();
  const int v = threadIdx.x;  // this thread's four columns
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  const bool has = v < hidden / 4;
  float g[4] = {}, bt[4] = {};
  if (has) {
    if (GB_FP32) {
      const float4 g4 = __ldg(reinterpret_cast<const float4*>(gamma) + v), b4 = __ldg(reinterpret_cast<const float4*>(beta) + v);
      g[0] = g4.x; g[1] = g4.y; g[2] = g4.z; g[3] = g4.w;
      bt[0] = b4.x; bt[1] = b4.y; bt[2] = b4.z; bt[3] = b4.w;
    } else {
      const uint2 g2 = __ldg(reinterpret_cast<const uint2*>(gamma) + v), b2 = __ldg(reinterpret_cast<const uint2*>(beta) + v);
      const float2 g0 = __half22float2(reinterpret_cast<const __half2*>(&g2)[0]), g1 = __half22float2(reinterpret_cast<const __half2*>(&g2)[1]);
      const float2 b0 = __half22float2(reinterpret_cast<const __half2*>(&b2)[0]), b1 = __half22float2(reinterpret_cast<const __half2*>(&b2)[1]);
      g[0] = g0.x; g[1] = g0.y; g[2] = g1.x; g[3] = g1.y;
      bt[0] = b0.x; bt[1] = b0.y; bt[2] = b1.x; bt[3] = b1.y;
    }
  }
  pdl_wait();
  const int row0 = static_cast<int>(blockIdx.x) * ROWS;
  uint2* o2 = reinterpret_cast<uint2*>(out + static_cast<size_t>(row0) * hidden) + v;
  int src[ROWS];  // row of x, or -1: a row of zeros, or -2: no such row
  int row_limit = m_rows;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    src[r] = (ROWS == 1 || row0 + r < m_rows) ? row0 + r : -2;
    if (RESTORE && (ROWS == 1 || src[r] >= 0)) {
      const int b = src[r] / S;
      const int i = src[r] - b * S;
      const int off = __ldg(batch_idx + b);
      src[r] = i < __ldg(batch_idx + b + 1) - off ? off + i : -1;
    }
  }
  if (!RESTORE && m_dev != nullptr) row_limit = __ldg(m_dev);
  if (RESTORE && ROWS == 1 && src[0] < 0) {
    if (has) *o2 = make_uint2(0u, 0u);
    return;
  }
  float4 a[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    a[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has && (ROWS == 1 || src[r] >= 0)) {
      const float4* xr = reinterpret_cast<const float4*>(x + static_cast<size_t>(src[r]) * hidden) + v;
      float4 p[SPLITS];
#pragma unroll
      for (int sp = 0; sp < SPLITS; ++sp)
        p[sp] = (sp == 0 || sp < split.n) ? __ldg(xr + sp * (split.stride / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
      a[r] = p[0];
#pragma unroll
      for (int sp = 1; sp < SPLITS; ++sp) {
        a[r].x += p[sp].x;
        a[r].y += p[sp].y;
        a[r].z += p[sp].z;
        a[r].w += p[sp].w;
      }
    }
  }
  // (the rows were read before their existence was known: they lie inside the allocation either way)
  if (!RESTORE) {
    if (row0 >= row_limit) return;
#pragma unroll
    for (int r = 1; r < ROWS; ++r)
      if (row0 + r >= row_limit) src[r] = -2;
  }
  if (has) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r) vals[r][v & 1][v >> 1] = a[r];
  }
  __syncthreads();
  // Statistics as layernorm_rows_kernel forms them: the same columns per lane in the same order, so that both forms give
  // the same bits.  One row per CTA: every warp forms them for itself; more: a warp per row.
  const int nvec = hidden >> 3;
  auto row_stats = [&](int r) {
    float val[NVEC][8];
    float sum = 0.f;
#pragma unroll
    for (int it = 0; it < NVEC; ++it) {
      const int u = it * 32 + lane;
      if (it + 1 < NVEC || u < nvec) {
        const float4 lo = vals[r][0][u], hi = vals[r][1][u];
        val[it][0] = lo.x; val[it][1] = lo.y; val[it][2] = lo.z; val[it][3] = lo.w;
        val[it][4] = hi.x; val[it][5] = hi.y; val[it][6] = hi.z; val[it][7] = hi.w;
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += val[it][k];
      }
    }
    const float mean = warp_sum(sum) / static_cast<float>(hidden);
    float sq = 0.f;
#pragma unroll
    for (int it = 0; it < NVEC; ++it) {
      if (it + 1 < NVEC || it * 32 + lane < nvec) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float d = val[it][k] - mean;
          sq = fmaf(d, d, sq);
        }
      }
    }
    return make_float2(mean, rsqrtf(warp_sum(sq) / static_cast<float>(hidden) + eps));
  };
  float2 st[ROWS];
  if (ROWS == 1) {
    st[0] = row_stats(0);
  } else {
    for (int r = warp; r < ROWS; r += n_warps) {
      const float2 t = row_stats(r);
      if (lane == 0) stats[r] = t;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROWS; ++r) st[r] = stats[r];
  }
  if (!has) return;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    if (ROWS > 1 && src[r] == -2) continue;
    const float mean = st[r].x, rstd = st[r].y;
    o2[r * (hidden / 4)] = (ROWS > 1 && src[r] < 0) ? make_uint2(0u, 0u)
                                      : make_uint2(pack_half2(fmaf((a[r].x - mean) * rstd, g[0], bt[0]),
                                                              fmaf((a[r].y - mean) * rstd, g[1], bt[1])),
                                                   pack_half2(fmaf((a[r].z - mean) * rstd, g[2], bt[2]),
                                                              fmaf((a[r].w - mean) * rstd, g[3], bt[3])));
  }
}

bool ln_cta_possible(const void* x, bool x_fp32, const __half* bias, const __half* residual, const void* gamma,
                     const void* beta) {
  return x_fp32 && bias == nullptr && residual == nullptr &&
         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta)) & 15u) == 0;
}
template <bool RESTORE, bool GB_FP32, int NVEC>
cudaError_t launch_ln_cta(const void* x, const void* gamma, const void* beta, __half* out, const int* m_dev, int rows,
                          const int* batch_idx, int S, int hidden, float eps, LnSplit split, int per_cta,
                          cudaStream_t stream) {
  const dim3 block((hidden / 4 + 31) / 32 * 32);
  auto go = [&](auto kern) {
    return launch_pdl(kern, dim3((rows + per_cta - 1) / per_cta), block, 0, stream, reinterpret_cast<const float*>(x), gamma,
                      beta, out, m_dev, rows, batch_idx, S, hidden, eps, split);
  };
  if constexpr (NVEC > 1) {
    if (per_cta == 4) return go(layernorm_cta_kernel<RESTORE, GB_FP32, 1, 4, NVEC>);
  }
  if constexpr (NVEC <= 3) {
    if (per_cta == 2) return go(layernorm_cta_kernel<RESTORE, GB_FP32, 1, 2, NVEC>);
  }
  if (per_cta != 1) return cudaErrorInvalidValue;
  if (split.n <= 1) return go(layernorm_cta_kernel<RESTORE, GB_FP32, 1, 1, NVEC>);
  if (split.n <= 2) return go(layernorm_cta_kernel<RESTORE, GB_FP32, 2, 1, NVEC>);
  if (split.n <= 4) return go(layernorm_cta_kernel<RESTORE, GB_FP32, 4, 1, NVEC>);
  return go(layernorm_cta_kernel<RESTORE, GB_FP32, kLnMaxSplit, 1, NVEC>);
}
template <bool RESTORE, typename... Args>
cudaError_t launch_ln_cta_dispatch(bool gb_fp32, int nvec, Args... args) {
  switch (nvec) {
    case 1: return gb_fp32 ? launch_ln_cta<RESTORE, true, 1>(args...) : launch_ln_cta<RESTORE, false, 1>(args...);
    case 2: return gb_fp32 ? launch_ln_cta<RESTORE, true, 2>(args...) : launch_ln_cta<RESTORE, false, 2>(args...);
    case 3: return gb_fp32 ? launch_ln_cta<RESTORE, true, 3>(args...) : launch_ln_cta<RESTORE, false, 3>(args...);
    case 4: return gb_fp32 ? launch_ln_cta<RESTORE, true, 4>(args...) : launch_ln_cta<RESTORE, false, 4>(args...);
    default: return cudaErrorInvalidValue;
  }
}

template <bool RESTORE, bool GB_FP32, bool X_FP32>
cudaError_t launch_ln_nvec(int nvec_needed, dim3 grid, cudaStream_t stream, const void* x, const __half* bias,
                           const __half* residual, const void* gamma, const void* beta, __half* out,
                           const int* m_dev, int m_rows, const int* batch_idx, int S, int hidden, float eps) {
#define BT_LN_CASE(NV)                                                                                        \
  case NV:                                                                                                    \
    return launch_pdl(layernorm_rows_kernel<RESTORE, GB_FP32, X_FP32, NV>, grid, dim3(kLnWarps * 32), 0, stream,  \
                      x, bias, residual, gamma, beta, out, m_dev, m_rows, batch_idx, S, hidden, eps);
  switch (nvec_needed) {
    BT_LN_CASE(1)
    BT_LN_CASE(2)
    BT_LN_CASE(3)
    BT_LN_CASE(4)
    default: return cudaErrorInvalidValue;
  }
#undef BT_LN_CASE
  return cudaGetLastError();
}

// x[row, :] = gelu(x[row, :] + bias), in place.  A thread owns one 16-byte column vector (its bias slice
// is read once) and walks down the rows, four rows per trip so that four loads are in flight; the exact-form
// GELU costs one special-function op per element (gelu_erf_fast).  blockIdx.x selects the column block,
// blockIdx.y the first row.
__global__ void __launch_bounds__(128)
add_bias_gelu_kernel(uint4* __restrict__ x, const uint4* __restrict__ bias, const int* __restrict__ m_dev,
                     int m_rows, int nvec, int gelu_kind) {
  pdl_launch_dependents();
  pdl_wait();
  int M = m_rows;
  if (m_dev != nullptr) {
    const int md = __ldg(m_dev);
    M = md < M ? md : M;
  }
  const int v = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
  if (v >= nvec) return;
  float b[8];
  unpack8(__ldg(bias + v), b);
  const int stride = static_cast<int>(gridDim.y);
  for (int r0 = static_cast<int>(blockIdx.y); r0 < M; r0 += 4 * stride) {
    uint4 in[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + u * stride;
      if (r < M) in[u] = x[static_cast<size_t>(r) * nvec + v];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + u * stride;
      if (r < M) {
        float f[8];
        unpack8(in[u], f);
        if (gelu_kind == BT_GELU_TANH) {
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = gelu_tanh(f[k] + b[k]);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = gelu_erf_fast(f[k] + b[k]);
        }
        x[static_cast<size_t>(r) * nvec + v] = pack8(f);
      }
    }
  }
}

__device__ __forceinline__ float exp2f_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Logits are laid out [nh, B, S, S] as in the reference (softmax.h:33: ((head*B + b)*S + i)*S); S <= 1024.
// VEC path (S % 8 == 0): a warp owns one (b, i) row of the mask and walks the nh heads' logits rows that
// share it, so the additive term (1 - mask) * -10000 is read and converted once per nh rows; the next
// head's row is requested before the current one is worked on.  Everything is in units of log2
// (exp(x) = 2^(x log2 e)): one special-function op per element.  The other path: one warp per logits row.
template <bool VEC, int NIT>
__global__ void __launch_bounds__(128)
masked_softmax_kernel(__half* __restrict__ logits, const __half* __restrict__ mask, int B, int nh, int S,
                      float scale) {
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * 4 + warp;
  if (VEC) {
    const long long mask_rows = static_cast<long long>(B) * S;
    if (row >= mask_rows) return;
    const int nvec = S / 8;
    const float scale_l2 = scale * 1.4426950408889634f;
    const long long head_stride = mask_rows * S;  // halves between the same (b, i) row of two heads
    __half* lp = logits + row * S;
    float add[NIT][8];
    uint4 raw[2][NIT];  // the rows of the next two heads, in flight
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int v = it * 32 + lane;
      if (v < nvec) {
        raw[0][it] = *(reinterpret_cast<const uint4*>(lp) + v);
        if (nh > 1) raw[1][it] = *(reinterpret_cast<const uint4*>(lp + head_stride) + v);
        float m[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(mask + row * S) + v), m);
#pragma unroll
        for (int k = 0; k < 8; ++k) add[it][k] = fmaf(m[k], 14426.950408889634f, -14426.950408889634f);
      }
    }
    for (int h = 0; h < nh; ++h, lp += head_stride) {
      float val[NIT][8];
      float mx = -INFINITY;
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const int v = it * 32 + lane;
        if (v < nvec) {
          unpack8(raw[0][it], val[it]);
          raw[0][it] = raw[1][it];
          if (h + 2 < nh) raw[1][it] = *(reinterpret_cast<const uint4*>(lp + 2 * head_stride) + v);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            val[it][k] = fmaf(val[it][k], scale_l2, add[it][k]);
            mx = fmaxf(mx, val[it][k]);
          }
        }
      }
      mx = warp_max(mx);
      float sum = 0.f;
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        if (it * 32 + lane < nvec) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            val[it][k] = exp2f_fast(val[it][k] - mx);
            sum += val[it][k];
          }
        }
      }
      const float inv = 1.0f / (warp_sum(sum) + 1e-6f);
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const int v = it * 32 + lane;
        if (v < nvec) {
#pragma unroll
          for (int k = 0; k < 8; ++k) val[it][k] *= inv;
          *(reinterpret_cast<uint4*>(lp) + v) = pack8(val[it]);
        }
      }
    }
  } else {
    const long long rows = static_cast<long long>(B) * nh * S;
    if (row >= rows) return;
    const int i = static_cast<int>(row % S);
    const int b = static_cast<int>((row / S) % B);
    __half* lp = logits + row * S;
    const __half* mp = mask + (static_cast<long long>(b) * S + i) * S;
    float val[32];
    float mx = -INFINITY;
#pragma unroll
    for (int it = 0; it < 32; ++it) {
      const int j = it * 32 + lane;
      if (j < S) {
        val[it] = fmaf(__half2float(lp[j]), scale, (1.0f - __half2float(mp[j])) * -10000.0f);
        mx = fmaxf(mx, val[it]);
      }
    }
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int it = 0; it < 32; ++it) {
      if (it * 32 + lane < S) {
        val[it] = __expf(val[it] - mx);
        sum += val[it];
      }
    }
    const float inv = 1.0f / (warp_sum(sum) + 1e-6f);
#pragma unroll
    for (int it = 0; it < 32; ++it) {
      const int j = it * 32 + lane;
      if (j < S) lp[j] = __float2half_rn(val[it] * inv);
    }
  }
}

}  // namespace

// at most 16 resident blocks (64 warps) per SM on 148 SMs
static unsigned ln_grid(long long blocks_needed) {
  const long long cap = 148LL * 16;
  return static_cast<unsigned>(blocks_needed < cap ? (blocks_needed < 1 ? 1 : blocks_needed) : cap);
}

template <bool RESTORE>
static cudaError_t launch_ln_dispatch(bool gb_fp32, bool x_fp32, int nv, dim3 grid, cudaStream_t stream, const void* x,
                                      const __half* bias, const __half* residual, const void* gamma, const void* beta,
                                      __half* out, const int* m_dev, int m_rows, const int* batch_idx, int S,
                                      int hidden, float eps) {
#define BT_LN_ARGS nv, grid, stream, x, bias, residual, gamma, beta, out, m_dev, m_rows, batch_idx, S, hidden, eps
  if (gb_fp32) {
    if (x_fp32) return launch_ln_nvec<RESTORE, true, true>(BT_LN_ARGS);
    return launch_ln_nvec<RESTORE, true, false>(BT_LN_ARGS);
  }
  if (x_fp32) return launch_ln_nvec<RESTORE, false, true>(BT_LN_ARGS);
  return launch_ln_nvec<RESTORE, false, false>(BT_LN_ARGS);
#undef BT_LN_ARGS
}

int ln_rows_per_cta(long long rows, int hidden, int parts, bool in_forward) {
  const long long sums = rows * hidden;
  if (hidden > kLnMaxVec * 256 || rows > 4096) return 0;
  if (!in_forward && hidden < 512 && rows > 512) return 0;
  if (rows <= 1024) return (parts <= 1 && hidden >= 512 && sums >= 400 * 768) ? 4 : 1;
  if (hidden >= 512 && hidden < 640 && rows <= 1536) return 2;
  if (hidden >= 512) return (in_forward || sums <= 2048 * 768) ? 4 : 0;
  return (in_forward && hidden >= 256) ? 2 : 0;
}

cudaError_t launch_layernorm(const void* x, bool x_fp32, const __half* bias, const __half* residual,
                             const void* gamma, const void* beta, bool gb_fp32, __half* out, const int* m_dev,
                             int m_rows, int hidden, float eps, cudaStream_t stream, LnSplit split) {
  if (hidden % 8 != 0 || hidden > kLnMaxVec * 256 || m_rows <= 0) return cudaErrorInvalidValue;
  if (split.n > 1 && (!x_fp32 || split.stride % 4 != 0 || split.n > kLnMaxSplit)) return cudaErrorInvalidValue;
  const int nv = (hidden / 8 + 31) / 32;
  const int per_cta = ln_rows_per_cta(m_rows, hidden, split.n, split.in_forward);
  if (per_cta != 0 && ln_cta_possible(x, x_fp32, bias, residual, gamma, beta))
    return launch_ln_cta_dispatch<false>(gb_fp32, nv, x, gamma, beta, out, m_dev, m_rows, static_cast<const int*>(nullptr), 0,
                                         hidden, eps, split, per_cta, stream);
  if (split.n > 1) return cudaErrorInvalidValue;  // partial sums come in calls of up to 1024 rows, from aligned buffers
  dim3 grid(ln_grid((m_rows + kLnWarps - 1) / kLnWarps));
  return launch_ln_dispatch<false>(gb_fp32, x_fp32, nv, grid, stream, x, bias, residual, gamma, beta, out, m_dev,
                                   m_rows, nullptr, 0, hidden, eps);
}

cudaError_t launch_layernorm_restore(const void* x, bool x_fp32, const __half* bias, const __half* residual,
                                     const void* gamma, const void* beta, bool gb_fp32, __half* out_padded,
                                     const int* batch_idx, int B, int S, int hidden, float eps,
                                     cudaStream_t stream, LnSplit split) {
  if (hidden % 8 != 0 || hidden > kLnMaxVec * 256 || B <= 0 || S <= 0) return cudaErrorInvalidValue;
  if (split.n > 1 && (!x_fp32 || split.stride % 4 != 0 || split.n > kLnMaxSplit)) return cudaErrorInvalidValue;
  const int nv = (hidden / 8 + 31) / 32;
  const long long rows = static_cast<long long>(B) * S;
  const int per_cta = ln_rows_per_cta(rows, hidden, split.n, split.in_forward);
  if (per_cta != 0 && ln_cta_possible(x, x_fp32, bias, residual, gamma, beta))
    return launch_ln_cta_dispatch<true>(gb_fp32, nv, x, gamma, beta, out_padded, static_cast<const int*>(nullptr),
                                        static_cast<int>(rows), batch_idx, S, hidden, eps, split, per_cta, stream);
  if (split.n > 1) return cudaErrorInvalidValue;
  dim3 grid(ln_grid((rows + kLnWarps - 1) / kLnWarps));
  return launch_ln_dispatch<true>(gb_fp32, x_fp32, nv, grid, stream, x, bias, residual, gamma, beta, out_padded,
                                  nullptr, static_cast<int>(rows), batch_idx, S, hidden, eps);
}

cudaError_t launch_add_bias_gelu(__half* x, const __half* bias, const int* m_dev, int m_rows, int n, int gelu_kind,
                                 cudaStream_t stream) {
  if (n % 8 != 0 || m_rows <= 0) return cudaErrorInvalidValue;
  const int nvec = n / 8;
  const unsigned gx = static_cast<unsigned>((nvec + 127) / 128);
  // enough row groups for ~16 CTAs per SM, never more than rows
  long long gy = (148LL * 16 + gx - 1) / gx;
  if (gy > m_rows) gy = m_rows;
  if (gy > 65535) gy = 65535;
  if (gy < 1) gy = 1;
  return launch_pdl(add_bias_gelu_kernel, dim3(gx, static_cast<unsigned>(gy)), dim3(128), 0, stream,
                    reinterpret_cast<uint4*>(x), reinterpret_cast<const uint4*>(bias), m_dev, m_rows, nvec, gelu_kind);
}

cudaError_t launch_masked_softmax(__half* logits, const __half* mask, int B, int nh, int S, float scale,
                                  cudaStream_t stream) {
  if (S <= 0 || S > 1024 || B <= 0 || nh <= 0) return cudaErrorInvalidValue;
  const long long rows = static_cast<long long>(B) * nh * S;
  if (S % 8 == 0) {  // a warp per mask row, looping over the heads
    dim3 grid_v(static_cast<unsigned>((static_cast<long long>(B) * S + 3) / 4));
    if (S <= 256) return launch_pdl(masked_softmax_kernel<true, 1>, grid_v, dim3(128), 0, stream, logits, mask, B, nh, S, scale);
    if (S <= 512) return launch_pdl(masked_softmax_kernel<true, 2>, grid_v, dim3(128), 0, stream, logits, mask, B, nh, S, scale);
    return launch_pdl(masked_softmax_kernel<true, 4>, grid_v, dim3(128), 0, stream, logits, mask, B, nh, S, scale);
  }
  dim3 grid(static_cast<unsigned>((rows + 3) / 4));
  return launch_pdl(masked_softmax_kernel<false, 4>, grid, dim3(128), 0, stream, logits, mask, B, nh, S, scale);
}

// ---------------------------------------------------------------------------------------
// Self-test of the bounded wait every pipeline of the library relies on: one CTA waits on an
// mbarrier that nothing will ever arrive on.  The wait must give up after `max_cycles`, record
// kStatusSelfTestTimeout in the status word and let the kernel return normally, leaving the
// context usable.  Nothing faults, traps or spins without a limit.
// ---------------------------------------------------------------------------------------
namespace {
__global__ void __launch_bounds__(64) bounded_wait_selftest_kernel(int* status, long long max_cycles, int* gave_up) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag_s;
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    abort_flag_s = 0;
    fence_mbar_init();
  }
  __syncthreads();
  volatile int* abort_flag = &abort_flag_s;
  if (threadIdx.x == 0) {
    // phase 0 never completes: no thread arrives on `bar`
    const bool got = mbar_wait_bounded(&bar, 0u, abort_flag, status, kStatusSelfTestTimeout, max_cycles);
    if (gave_up != nullptr) *gave_up = got ? 0 : 1;
  } else if (threadIdx.x == 32) {
    // a second role that sees the first one give up through the CTA's abort flag
    long long spins = 0;
    while (*abort_flag == 0 && spins < max_cycles) spins += 64, __nanosleep(64);
  }
  __syncthreads();
}

// A K loop's waits after one of them gave up: 64 waits for a barrier that nothing arrives on.  out[0] = clocks of
// the first, out[1] = of all, out[2] = lanes that believe a wait succeeded.  out[3] = lanes told so by a warp's wait
// where one lane's barrier has completed its phase and the others' has not.
__global__ void __launch_bounds__(32) wait_forms_selftest_kernel(long long max_cycles, long long* out) {
  __shared__ uint64_t bar, done;
  __shared__ int abort_flag_s;
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_init(&done, 1);
    abort_flag_s = 0;
    fence_mbar_init();
    mbar_arrive(&done);
  }
  __syncthreads();
  const long long t0 = clock64();
  bool ok = true;
  long long t1 = t0;
  for (int kb = 0; kb < 64; ++kb) {
    ok = mbar_wait_latched(ok, false, &bar, 0u, &abort_flag_s, nullptr, 0, max_cycles);
    if (kb == 0) t1 = clock64();
  }
  const long long t2 = clock64();
  const int lanes = __popc(__ballot_sync(0xffffffffu, ok));
  abort_flag_s = 0;
  __syncwarp();
  const bool got = mbar_wait_warp(threadIdx.x == 5 ? &done : &bar, 0u, &abort_flag_s, nullptr, 0, max_cycles);
  const int told = __popc(__ballot_sync(0xffffffffu, got));
  if (threadIdx.x == 0) {
    out[0] = t1 - t0;
    out[1] = t2 - t0;
    out[2] = lanes;
    out[3] = told;
  }
}
// accumulators_back after three tiles (buffer 0 handed back twice, buffer 1 once).  out[k] = lanes told that tensor memory
// may go: k = 0 all came, 1 all came and the flag is up, 2 the last one of buffer 0 is missing, 3 no tile was begun.
__global__ void __launch_bounds__(32) accumulators_back_selftest_kernel(long long max_cycles, long long* out) {
  __shared__ uint64_t acc[2], late[2];
  __shared__ int abort_flag_s;
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc[i], 1);
      mbar_init(&late[i], 1);
    }
    abort_flag_s = 0;
    fence_mbar_init();
    for (int it = 0; it < 3; ++it) mbar_arrive(&acc[it & 1]);
    for (int it = 0; it < 2; ++it) mbar_arrive(&late[it & 1]);
  }
  __syncthreads();
  for (int k = 0; k < 4; ++k) {
    abort_flag_s = k == 1 ? 1 : 0;
    __syncwarp();
    const bool may_go = accumulators_back(k == 2 ? late : acc, k == 3 ? 0 : 3, &abort_flag_s, nullptr, 0, max_cycles);
    const int told = __popc(__ballot_sync(0xffffffffu, may_go));
    if (threadIdx.x == 0) out[k] = told;
    __syncwarp();
  }
}
}  // namespace

cudaError_t launch_bounded_wait_selftest(int* status, long long max_cycles, int* gave_up, cudaStream_t stream) {
  if (max_cycles < 1024) max_cycles = 1024;
  if (max_cycles > (1ll << 31)) max_cycles = (1ll << 31);
  return launch_pdl(bounded_wait_selftest_kernel, dim3(1), dim3(64), 0, stream, status, max_cycles, gave_up);
}

static cudaError_t launch_wait_forms_selftest(long long max_cycles, long long* out, cudaStream_t stream) {
  if (max_cycles < 1024) max_cycles = 1024;
  if (max_cycles > (1ll << 28)) max_cycles = (1ll << 28);
  return launch_pdl(wait_forms_selftest_kernel, dim3(1), dim3(32), 0, stream, max_cycles, out);
}

static cudaError_t launch_accumulators_back_selftest(long long max_cycles, long long* out, cudaStream_t stream) {
  if (max_cycles < 1024) max_cycles = 1024;
  if (max_cycles > (1ll << 28)) max_cycles = (1ll << 28);
  return launch_pdl(accumulators_back_selftest_kernel, dim3(1), dim3(32), 0, stream, max_cycles, out);
}

}  // namespace bt

// Diagnostics hook (tests): see accumulators_back_selftest_kernel; `out_dev` holds four long long.
extern "C" int bt_debug_selftest_accumulators_back(long long max_cycles, long long* out_dev, void* stream) {
  if (out_dev == nullptr) return BT_ERR_INVALID_ARG;
  return bt::launch_accumulators_back_selftest(max_cycles, out_dev, reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess
             ? BT_OK : BT_ERR_CUDA;
}

// Diagnostics hook (tests): see wait_forms_selftest_kernel; `out_dev` holds four long long.
extern "C" int bt_debug_selftest_wait_forms(long long max_cycles, long long* out_dev, void* stream) {
  if (out_dev == nullptr) return BT_ERR_INVALID_ARG;
  return bt::launch_wait_forms_selftest(max_cycles, out_dev, reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess
             ? BT_OK : BT_ERR_CUDA;
}
