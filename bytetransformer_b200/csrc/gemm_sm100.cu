// Dense fp16 GEMM for sm_100a:  out[M,N] = epilogue(A[M,K] * W[K,N]),  fp32 accumulation.
//
// Replaces the reference's cuBLAS / CUTLASS-2.x calls on the encoder path
// (bytetransformer/src/gemm.cu:32-39, bytetransformer/src/gemm_bias_act.cu:76-148).
//
// Two persistent kernels share one epilogue:
//
//  gemm_f16_kernel<BLOCK_N, EPI>      one CTA per SM, tile 128 x BLOCK_N (256/128/64),
//                                     tcgen05.mma.cta_group::1.
//  gemm_f16_pair_kernel<EPI>          clusters of two CTAs on an SM pair, tile 256 x 256:
//                                     each CTA loads its 128 rows of A and HALF of the W
//                                     tile (128 of the 256 columns); the leader CTA issues
//                                     tcgen05.mma.cta_group::2 (M = 256), which feeds both
//                                     SMs' tensor cores from the two halves.  Per SM this
//                                     halves the shared-memory fill and the L2 traffic of
//                                     W and makes room for a 6-stage ring.  Used whenever
//                                     the problem has enough 256-row tiles.
//
// Roles in every CTA (320 threads):
//   warp 0      TMA producer: A tile [128 x 64] (K-major) and W tile [64 x n] (N contiguous
//               = MN-major for UMMA, so the reference's [in,out] weight layout is consumed
//               as is, no transposed copy) into a 128B-swizzled shared-memory ring.
//   warp 1      allocates tensor memory and (leader only, for the pair kernel) issues the
//               MMAs (the warp walks the loop, an elected lane's instructions take effect: see
//               common.cuh); accumulators are double buffered in tensor memory
//               (2 x 256 columns) so the epilogue of tile i overlaps the main loop of i+1.
//   warps 2..9  epilogue: tcgen05.ld -> +bias -> GELU / +residual -> fp16 (or fp32)
//               -> 128B-swizzled staging rows in shared memory -> TMA bulk store
//               (full 128-byte lines); a 32-row slab that crosses M falls back to
//               row-predicated 16-byte stores, so rows >= M are never written.
// M is read from device memory (the packed token count is only known on the device), so
// the host never blocks; the grid is sized from the allocated rows.  Every mbarrier wait
// is bounded: on expiry the CTA records a code in the status word and all roles drain to
// a common exit that frees tensor memory.  (The one-CTA kernels free it ahead of the exit where
// no wait has run out: see accumulators_back.)  No TMA load uses cluster multicast.
#include "common.cuh"
#include "kernels.h"
#include "../../include/bt_b200.h"

namespace bt {

namespace {

constexpr int kBlockM = 128;
constexpr int kBlockK = 64;
constexpr int kGemmThreads = 320;
constexpr int kEpiWarps = 8;
constexpr int kABytes = kBlockM * kBlockK * 2;  // 16 KiB
constexpr int kStagingBytesPerWarp = 32 * 128;  // 32 rows x 128 B
constexpr int kBarBytes = 256;                  // barriers, tensor memory address, flag
// Every epilogue warp's own copy of the bias of its columns, half of a tile's: see BiasShare.
constexpr int bias_bytes(int tile_n) { return kEpiWarps * (tile_n / 2) * 2; }

template <int BLOCK_N>
struct GemmCfg {
  static constexpr int kBBytes = BLOCK_N * kBlockK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = (BLOCK_N == 256) ? 4 : (BLOCK_N == 128 ? 6 : 8);
  static constexpr int kTmemCols = 2 * BLOCK_N;
  // Output leaves through per-warp staging rows + TMA bulk stores when a warp's column share of a row is at
  // least 128 bytes: 64 fp16 or 32 fp32 columns.
  static constexpr bool tma_store(int epi) {
    return BLOCK_N >= 128 || epi == BT_EPI_BIAS_RESIDUAL_F32OUT || epi == kEpiSplitKF32;
  }
  static constexpr int kStagingBytes = kEpiWarps * kStagingBytesPerWarp;
  static constexpr int kSmemBytes = kStages * kStageBytes + kStagingBytes + kBarBytes + bias_bytes(BLOCK_N);
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of the one-CTA GEMM kernel");
};

// Pair kernel: per CTA 128 rows of A and 128 of the tile's 256 W columns per stage.
struct PairCfg {
  static constexpr int kTileN = 256;
  static constexpr int kBHalfBytes = 128 * kBlockK * 2;  // 16 KiB
  static constexpr int kStageBytes = kABytes + kBHalfBytes;
  static constexpr int kStages = 6;
  static constexpr int kTmemCols = 512;
  static constexpr int kStagingBufs = 1;  // per epilogue warp (two were measured: no gain, and they cost a stage)
  static constexpr int kStagingBytes = kStagingBufs * kEpiWarps * kStagingBytesPerWarp;
  static constexpr int kSmemBytes = kStages * kStageBytes + kStagingBytes + kBarBytes + bias_bytes(kTileN);
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of the SM-pair GEMM kernel");
};

struct GemmArgs {
  __half* out;
  const __half* bias;
  const __half* residual;
  const int* m_dev;
  int m_rows;
  int N;
  int K;
  int* status;
  // fused LayerNorm (BT_EPI_BIAS_RESIDUAL_LAYERNORM): `out` is the scratch for the row
  // statistics partials (up to 16 * N/128 bytes per row), `out_ln` the fp16 result
  __half* out_ln;
  const void* gamma;
  const void* beta;
  int gb_fp32;
  float eps;
  uint32_t ln_epoch;  // fused LayerNorm: tag of this launch in the statistics scratch (see gemm_f16_ln_kernel)
  // split-K (kEpiSplitKF32): K is cut into `split_k` ranges, range s writes its fp32 partial sum to
  // out + s * split_stride floats; range 0 also adds bias and residual
  int split_k;
  long long split_stride;
  int early_w;  // request the first tile's W blocks before the wait for the kernel before
  int force_n;  // fused LayerNorm, diagnostics: tile width (0 = ln_tile_n)
  long long* timing;  // diagnostics: clock64 stamps per CTA and tile (null = off)
  uint64_t a_desc_hi;
  uint64_t b_desc_hi;
  uint32_t a_kstep_bytes;
  uint32_t b_kstep_bytes;
  uint32_t idesc;
};

// Debug overrides (0 = default): W descriptor fields, forced tile width, pair kernel on/off.
long long* g_dbg_gemm_timing = nullptr;  // [148 CTAs][16 tiles][8 slots]
__device__ __forceinline__ void gstamp(long long* timing, int it, int slot) {
  if (timing != nullptr && it < 16 && blockIdx.x < 148) timing[(blockIdx.x * 16 + it) * 8 + slot] = clock64();
}
long long g_dbg_b_lbo = 0, g_dbg_b_sbo = 0, g_dbg_b_kstep = 0, g_dbg_force_block_n = 0, g_dbg_pair_mode = 0;
long long g_dbg_early_w = 1;  // 1 = W blocks of the first tile requested before the dependency wait
long long g_dbg_ln_pair = 0;  // GEMM + LayerNorm on SM pairs: 0 = by ln_pair_pays (default), 1 = always, anything else = never
long long g_dbg_split_k = 0;  // 0 = policy, < 0 = never, > 0 = that many ranges whenever the shape allows

// ------------------------------------------------------------------------------------------
// Epilogue of one 128 x TILE_N accumulator tile, executed by the 8 epilogue warps of a CTA.
// The warp owns TMEM lanes (warp_id % 4) * 32 .. +31 (`quarter`) and one half of the tile's
// columns (`col_half`).  `tm_out` is the store map (box 128 B x 32 rows).
// ------------------------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void tma_store_wait_read_n() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

// STG_BUFS staging buffers of 32 rows x 128 B per warp are used in turn, so a bulk store
// only has to wait for the store issued STG_BUFS chunks earlier.  The accumulator chunk
// c+1 is requested from tensor memory before chunk c is processed.
template <int TILE_N, int EPI, bool TMA_STORE, int STG_BUFS>
__device__ __forceinline__ void epilogue_tile(const GemmArgs& args, const CUtensorMap* tm_out, uint8_t* stg,
                                              uint32_t tmem_acc, int m0, int n0, int M, int quarter, int col_half,
                                              int lane, const uint4* resv, const uint4* bias_s, int split = 0) {
  constexpr int kColsPerWarp = TILE_N / 2;
  constexpr bool kSplitK = (EPI == kEpiSplitKF32);
  constexpr bool kF32Out = (EPI == BT_EPI_BIAS_RESIDUAL_F32OUT) || kSplitK;
  constexpr bool kHasResidual = (EPI == BT_EPI_BIAS_RESIDUAL || EPI == BT_EPI_BIAS_RESIDUAL_F32OUT) || kSplitK;
  // 128 bytes of output per row and chunk: 32 fp32 or 64 fp16 columns.
  constexpr int kChunk = kF32Out ? 32 : (kColsPerWarp >= 64 ? 64 : 32);
  constexpr int kNChunks = kColsPerWarp / kChunk;
  constexpr int kHalves = kChunk / 32;  // tcgen05.ld x32 per chunk
  const int row0 = m0 + quarter * 32;
  const int row = row0 + lane;
  const bool row_ok = row < M;
  const bool slab_full = TMA_STORE && (row0 + 32 <= M);  // all 32 rows valid: bulk store, else predicated stores
  const uint32_t t_row = tmem_acc + (static_cast<uint32_t>(quarter * 32) << 16) + col_half * kColsPerWarp;
  uint32_t raw[2][kHalves][32];
#pragma unroll
  for (int h = 0; h < kHalves; ++h) tmem_ld_32x32(t_row + h * 32, raw[0][h]);
  tmem_ld_wait();
#pragma unroll
  for (int ci = 0; ci < kNChunks; ++ci) {
    const int c = ci * kChunk;
    const int col = col_half * kColsPerWarp + c;  // column inside the tile
    const int gcol = n0 + col;
    if (ci + 1 < kNChunks) {
#pragma unroll
      for (int h = 0; h < kHalves; ++h) tmem_ld_32x32(t_row + c + kChunk + h * 32, raw[(ci + 1) & 1][h]);
    }
    float v[kChunk];
#pragma unroll
    for (int h = 0; h < kHalves; ++h)
#pragma unroll
      for (int i = 0; i < 32; ++i) v[h * 32 + i] = __uint_as_float(raw[ci & 1][h][i]);
    if (EPI != BT_EPI_NONE && (!kSplitK || split == 0)) {
#pragma unroll
      for (int q = 0; q < kChunk / 8; ++q) {
        const uint4 b4 = bias_s[c / 8 + q];
        const uint32_t bh[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) add_half2(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1], bh[j]);
      }
    }
    // (Two instances, not a branch: with both forms in one kernel a 128 x 256 tile's epilogue took 5.7k clocks, by
    // itself the erf form takes 4.85k; tile period of 18,944 x 3072 x 768 7.35k / 6.9k.)
    if (EPI == BT_EPI_BIAS_GELU) {
#pragma unroll
      for (int i = 0; i < kChunk; i += 2) gelu_erf_fast_pair(v[i], v[i + 1]);
    } else if (EPI == kEpiBiasGeluTanh) {
#pragma unroll
      for (int i = 0; i < kChunk; ++i) v[i] = gelu_tanh(v[i]);
    }
    const size_t off = static_cast<size_t>(row) * args.N + gcol +
                       (kSplitK ? static_cast<size_t>(split) * static_cast<size_t>(args.split_stride) : 0);
    if (kHasResidual) {
#pragma unroll
      for (int q = 0; q < kChunk / 8; ++q) {
        const uint4 r4 = resv[c / 8 + q];
        const uint32_t rh[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) add_half2(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1], rh[j]);
      }
    }
    // 8 (or 4) units of 16 bytes per row
    constexpr int kUnits = kF32Out ? 8 : kChunk / 8;
    uint4 units[kUnits];
    if (kF32Out) {
#pragma unroll
      for (int q = 0; q < 8; ++q)
        units[q] = make_uint4(__float_as_uint(v[q * 4]), __float_as_uint(v[q * 4 + 1]), __float_as_uint(v[q * 4 + 2]),
                              __float_as_uint(v[q * 4 + 3]));
    } else {
#pragma unroll
      for (int q = 0; q < kChunk / 8; ++q) {
        units[q].x = pack_half2(v[q * 8 + 0], v[q * 8 + 1]);
        units[q].y = pack_half2(v[q * 8 + 2], v[q * 8 + 3]);
        units[q].z = pack_half2(v[q * 8 + 4], v[q * 8 + 5]);
        units[q].w = pack_half2(v[q * 8 + 6], v[q * 8 + 7]);
      }
    }
    if (slab_full) {
      // the bulk store that last used this staging buffer must have finished reading it
      if (lane == 0) tma_store_wait_read_n<STG_BUFS - 1>();
      __syncwarp();
      uint8_t* sbuf = stg + (STG_BUFS == 2 ? (ci & 1) * kStagingBytesPerWarp : 0);
      uint8_t* srow = sbuf + lane * 128;
#pragma unroll
      for (int q = 0; q < kUnits; ++q) *reinterpret_cast<uint4*>(srow + ((q ^ (lane & 7)) << 4)) = units[q];
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        // (the partial sums of a split lie below one another in the store map: split_stride = m_rows * N)
        tma_store_2d(tm_out, sbuf, gcol, kSplitK ? split * args.m_rows + row0 : row0);
        tma_store_commit();
      }
    } else if (row_ok) {
      uint4* op = kF32Out ? reinterpret_cast<uint4*>(reinterpret_cast<float*>(args.out) + off)
                          : reinterpret_cast<uint4*>(args.out + off);
#pragma unroll
      for (int q = 0; q < kUnits; ++q) op[q] = units[q];
    }
    if (ci + 1 < kNChunks) tmem_ld_wait();
  }
}

// The residual slice of a thread's row, fetched before the accumulator is waited for so that
// its latency hides behind the main loop of the tile.
template <int TILE_N, int EPI>
__device__ __forceinline__ void prefetch_residual(const GemmArgs& args, int m0, int n0, int M, int quarter,
                                                  int col_half, int lane, uint4* resv, int split = 0) {
  constexpr int kColsPerWarp = TILE_N / 2;
  constexpr bool kHasResidual = (EPI == BT_EPI_BIAS_RESIDUAL || EPI == BT_EPI_BIAS_RESIDUAL_F32OUT ||
                                 EPI == BT_EPI_BIAS_RESIDUAL_LAYERNORM || EPI == kEpiSplitKF32);
  if (kHasResidual) {
    const int row = m0 + quarter * 32 + lane;
    const bool row_ok = row < M && split == 0;  // only the first K range carries the residual
    const uint4* rp = reinterpret_cast<const uint4*>(args.residual + static_cast<size_t>(row) * args.N + n0 +
                                                     col_half * kColsPerWarp);
#pragma unroll
    for (int q = 0; q < kColsPerWarp / 8; ++q) resv[q] = row_ok ? __ldg(rp + q) : make_uint4(0u, 0u, 0u, 0u);
  }
}

// The bias of a warp's columns: asked for before the accumulator is waited for (BiasShare holds the lane's share), then put
// where the warp reads it column by column - read from global memory there, a chunk's loads took a round trip to L2 in
// the middle of the epilogue.  Each warp has a place of its own (bias_slice), so that nothing but its own __syncwarp orders
// one tile's reads before the next tile's writes: the hand-back of an accumulator to the MMAs orders no memory.
template <int TILE_N>
__device__ __forceinline__ __half* bias_slice(uint64_t* bars, int epi_warp) {
  return reinterpret_cast<__half*>(reinterpret_cast<uint8_t*>(bars) + kBarBytes) + epi_warp * (TILE_N / 2);
}
template <int TILE_N>
struct BiasShare {
  static constexpr int kPerLane = TILE_N / 64;  // halves
  alignas(8) __half v[kPerLane];
  __device__ __forceinline__ void load(const __half* bias, int n0, int col_half, int lane) {
    const __half* p = bias + n0 + col_half * (TILE_N / 2) + lane * kPerLane;
    if (kPerLane == 4)
      *reinterpret_cast<uint2*>(v) = __ldg(reinterpret_cast<const uint2*>(p));
    else if (kPerLane == 2)
      *reinterpret_cast<uint32_t*>(v) = __ldg(reinterpret_cast<const uint32_t*>(p));
    else
      v[0] = __ldg(p);
  }
  // (called by the whole warp, whose reads of the tile before are behind a __syncwarp)
  __device__ __forceinline__ void put(__half* bias_s, int lane) const {
    __half* p = bias_s + lane * kPerLane;
    if (kPerLane == 4)
      *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(v);
    else if (kPerLane == 2)
      *reinterpret_cast<uint32_t*>(p) = *reinterpret_cast<const uint32_t*>(v);
    else
      p[0] = v[0];
    __syncwarp();
  }
};

// Whether dynamic shared memory starts on the 1,024 bytes that the 128-byte swizzle needs, as it is declared to (there is
// no room to round up).  If not, the launch computes nothing and the status word says so.
__device__ __forceinline__ bool smem_aligned(const GemmArgs& args, const uint8_t* smem) {
  const bool ok = (smem_u32(smem) & 1023u) == 0u;
  if (!ok && threadIdx.x == 0 && args.status != nullptr) atomicCAS(args.status, 0, kStatusGemmProducerTimeout + 0x10);
  return ok;
}

// Rounds the start of shared memory up to where it is already (see smem_aligned).  Not for the address: formed this way
// the compiler keeps the kernels' shared-memory addresses in another form.  us per forward without / with: 38 tokens, 12
// layers 344.1 / 338.2; SM-pair kernel, 16 x 512 causal 1702 / 1675, 64 x 384 with 24 layers 9252 / 9143.
__device__ __forceinline__ uint8_t* round_up_1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// ------------------------------------------------------------------------------------------
// One CTA per SM, tile 128 x BLOCK_N.
// ------------------------------------------------------------------------------------------
template <int BLOCK_N, int EPI>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                const __grid_constant__ CUtensorMap tm_out, const GemmArgs args) {
  using Cfg = GemmCfg<BLOCK_N>;
  constexpr int kStages = Cfg::kStages;
  constexpr bool kSplitK = (EPI == kEpiSplitKF32);
  constexpr bool kHasResidual = (EPI == BT_EPI_BIAS_RESIDUAL || EPI == BT_EPI_BIAS_RESIDUAL_F32OUT) || kSplitK;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const bool smem_ok = smem_aligned(args, smem_raw);
  uint8_t* smem = round_up_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes + Cfg::kStagingBytes);
  uint64_t* full_bar = bars;                    // [kStages]
  uint64_t* empty_bar = bars + kStages;         // [kStages]
  uint64_t* acc_full = bars + 2 * kStages;      // [2]
  uint64_t* acc_empty = bars + 2 * kStages + 2; // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_int(static_cast<int>(threadIdx.x >> 5));  // warp-uniform roles: see common.cuh
  const int lane = threadIdx.x & 31;

  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], kEpiWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
    tma_prefetch_desc(&tm_out);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform_u32(*tmem_slot);

  const int n_tiles = args.N / BLOCK_N;
  const int splits = kSplitK ? args.split_k : 1;
  const int num_kb = args.K / kBlockK / splits;  // K blocks per tile (per K range with split-K)
  // Tile number -> (K range, column block, row block).  The K range and the column block come from
  // the low part of the number, so those of a CTA's first tile (number blockIdx.x) are known before
  // the row count is.
  auto tile_cols = [&](int tile, int& n0, int& sp) -> int {
    sp = 0;
    if (kSplitK) {
      sp = tile % splits;
      tile /= splits;
    }
    n0 = (tile % n_tiles) * BLOCK_N;
    return tile / n_tiles;
  };
  // The weights are written by no kernel of the chain, so the W blocks of the first tile are
  // requested before the wait for the kernel before (whose tail they then overlap): the first
  // `pre_kb` stages get their full byte count armed and their W part requested here, their A
  // part after the wait.
  const int pre_kb = args.early_w && smem_ok ? (num_kb < kStages ? num_kb : kStages) : 0;
  if (warp == 0) {
    int n0 = 0, sp = 0;
    tile_cols(static_cast<int>(blockIdx.x), n0, sp);
    for (int kb = 0; kb < pre_kb; ++kb) {
      uint8_t* sb = smem + kb * Cfg::kStageBytes + kABytes;
      if (elect_one()) mbar_arrive_expect_tx(&full_bar[kb], Cfg::kStageBytes);
#pragma unroll
      for (int c = 0; c < BLOCK_N / 64; ++c)
        if (elect_one()) tma_load_2d(sb + c * (64 * kBlockK * 2), &tm_b, &full_bar[kb], n0 + c * 64, (sp * num_kb + kb) * kBlockK);
    }
  } else if (warp >= 2 && EPI != BT_EPI_NONE && args.early_w && args.bias != nullptr) {
    // the bias slice of the first tile, for the same reason
    int n0 = 0, sp = 0;
    tile_cols(static_cast<int>(blockIdx.x), n0, sp);
    const __half* bp = args.bias + n0 + ((warp - 2) >> 2) * (BLOCK_N / 2);
    if (lane * 64 < BLOCK_N / 2) prefetch_l1(bp + lane * 64);
  }

  // Everything above touched only this CTA's own resources and the weights; from here on global
  // memory written by earlier kernels is read.  The A blocks of the armed stages go first, before
  // the row count is known: the first tile's rows lie inside the allocation whether or not they
  // are valid, and a CTA that turns out to have no tile only has to wait for them.
  pdl_wait();
  if (warp == 0 && pre_kb > 0) {
    int n0 = 0, sp = 0;
    const int m0 = tile_cols(static_cast<int>(blockIdx.x), n0, sp) * kBlockM;
    for (int kb = 0; kb < pre_kb; ++kb)
      if (elect_one()) tma_load_2d(smem + kb * Cfg::kStageBytes, &tm_a, &full_bar[kb], (sp * num_kb + kb) * kBlockK, m0);
  }
  int M = args.m_rows;
  if (args.m_dev != nullptr) {
    const int md = __ldg(args.m_dev);
    M = uniform_int(md < M ? md : M);
  }
  if (!smem_ok) M = 0;
  const int m_tiles = (M + kBlockM - 1) / kBlockM;
  const int total_tiles = m_tiles * n_tiles * splits;
  // The li-th tile of this CTA: tiles go round-robin over the CTAs.  With split-K a tile is an
  // (output tile, K range) pair; `sp` is the range.
  auto tile_at = [&](int li, int& m0, int& n0, int& sp) -> bool {
    const int tile = static_cast<int>(blockIdx.x) + li * static_cast<int>(gridDim.x);
    if (tile >= total_tiles) return false;
    m0 = tile_cols(tile, n0, sp) * kBlockM;
    return true;
  };
  bool tmem_freed = false;  // (warp 1's answer)

  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer
    {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int m0 = 0, n0 = 0, sp = 0;
      if (!tile_at(0, m0, n0, sp)) {
        // No tile for this CTA after all (fewer valid rows than allocated): wait for the armed
        // stages, so that no copy is in flight at exit.
        for (int kb = 0; kb < pre_kb; ++kb)
          if (!mbar_wait_warp(&full_bar[kb], 0u, abort_flag, args.status, kStatusGemmProducerTimeout)) break;
      }
      for (int li = 0; ok && tile_at(li, m0, n0, sp); ++li) {
        for (int i = 0; i < num_kb; ++i) {
          const int kb = sp * num_kb + i;
          uint8_t* sa = smem + stage * Cfg::kStageBytes;
          uint8_t* sb = sa + kABytes;
          if (li == 0 && i < pre_kb) {
            // armed and requested above (stage == i here)
          } else {
            if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1u, abort_flag, args.status,
                                   kStatusGemmProducerTimeout)) {
              ok = false;
              break;
            }
            if (elect_one()) mbar_arrive_expect_tx(&full_bar[stage], Cfg::kStageBytes);
            if (elect_one()) tma_load_2d(sa, &tm_a, &full_bar[stage], kb * kBlockK, m0);
#pragma unroll
            for (int c = 0; c < BLOCK_N / 64; ++c)
              if (elect_one()) tma_load_2d(sb + c * (64 * kBlockK * 2), &tm_b, &full_bar[stage], n0 + c * 64, kb * kBlockK);
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // --------------------------------------------------------------- MMA issuer
    {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true, landed = false;
      int m0 = 0, n0 = 0, sp = 0, tiles = 0;
      for (int it = 0; ok && tile_at(it, m0, n0, sp); ++it) {
        const int as = it & 1;
        const uint32_t aphase = (it >> 1) & 1;
        if (!mbar_wait_warp(&acc_empty[as], aphase ^ 1u, abort_flag, args.status, kStatusGemmMmaTimeout)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (lane == 0) gstamp(args.timing, it, 0);
        const uint32_t d_tmem = tmem_base + as * BLOCK_N;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_latched(ok, landed, &full_bar[stage], phase, abort_flag, args.status, kStatusGemmMmaTimeout);
          tc_fence_after();
          const int cur = stage;
          const uint32_t sa = smem_u32(smem + cur * Cfg::kStageBytes);
          const uint32_t sb = sa + kABytes;
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
          landed = mbar_test_wait(&full_bar[stage], phase);  // the next block, ahead of these MMAs
          // (the commit frees the stage once these MMAs have retired)
          umma_k_block<false>(d_tmem, smem_desc(args.a_desc_hi, sa), smem_desc(args.b_desc_hi, sb), args.a_kstep_bytes >> 4,
                       args.b_kstep_bytes >> 4, args.idesc, kb != 0 ? 1u : 0u, &empty_bar[cur]);
        }
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (ok && elect_one()) umma_commit(&acc_full[as]);
        if (lane == 0) gstamp(args.timing, it, 1);
        tiles = it + 1;
      }
      // Tensor memory goes back as soon as the accumulators have: at the end of the CTA it took 0.6k clocks of the
      // chain of kernels.
      if (accumulators_back(acc_empty, tiles, abort_flag, args.status, kStatusGemmMmaTimeout)) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
        tmem_freed = true;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int e = warp - 2;
    const int quarter = warp & 3;  // TMEM lane quarter this warp may read
    const int col_half = e >> 2;   // which half of the tile's columns
    uint8_t* stg = smem + kStages * Cfg::kStageBytes + e * kStagingBytesPerWarp;  // 32 rows x 128 B, swizzled
    __half* bias_s = bias_slice<BLOCK_N>(bars, e);
    int m0 = 0, n0 = 0, sp = 0;
    for (int it = 0; tile_at(it, m0, n0, sp); ++it) {
      const int as = it & 1;
      const uint32_t aphase = (it >> 1) & 1;
      uint4 resv[kHasResidual ? BLOCK_N / 16 : 1];
      prefetch_residual<BLOCK_N, EPI>(args, m0, n0, M, quarter, col_half, lane, resv, sp);
      BiasShare<BLOCK_N> bias;
      if (EPI != BT_EPI_NONE) bias.load(args.bias, n0, col_half, lane);
      mbar_wait_anyway(&acc_full[as], aphase, abort_flag, args.status, kStatusGemmEpilogueTimeout);
      tc_fence_after();
      if (EPI != BT_EPI_NONE) bias.put(bias_s, lane);
      if (warp == 2 && lane == 0) gstamp(args.timing, it, 2);
      epilogue_tile<BLOCK_N, EPI, Cfg::tma_store(EPI), 1>(args, &tm_out, stg, tmem_base + as * BLOCK_N, m0, n0, M, quarter,
                                                  col_half, lane, resv, reinterpret_cast<const uint4*>(bias_s), sp);
      if (warp == 2 && lane == 0) gstamp(args.timing, it, 3);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[as]);
    }
    if (Cfg::tma_store(EPI) && lane == 0) tma_store_wait_all();  // staging rows must outlive the last bulk store
  }

  // ------------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag != 0) {
    // A wait ran out somewhere: give copies and MMAs that may still be in flight time to
    // land before the CTA's shared and tensor memory are handed to another block.
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    if (warp == 1 && !tmem_freed) {  // (what kept it from being freed raised the flag)
      tc_fence_after();
      tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
  }
}

// ------------------------------------------------------------------------------------------
// Two CTAs per cluster (an SM pair), tile 256 x 256, tcgen05.mma.cta_group::2.
// CTA rank r of the pair owns rows m0 + r*128 .. +127 (its own accumulator in its own tensor
// memory) and stages W columns n0 + r*128 .. +127.  Barriers:
//   full[s]      leader's copy only: 1 arrival (leader's expect_tx of BOTH CTAs' bytes); the
//                peer's TMA completes its bytes on the leader's barrier.
//   empty[s]     one per CTA, arrived by the leader's commit multicast to both CTAs.
//   acc_full[a]  one per CTA, same multicast commit.
//   acc_empty[a] leader's copy only: 16 arrivals (8 epilogue warps of each CTA).
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t cta_rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(cta_rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Hands an accumulator buffer back to the leader.  Relaxed: what the MMAs wait for is that reads of tensor memory are
// done (tcgen05.wait::ld and the fences around the barrier); no bytes in memory go with it (what an epilogue warp keeps in
// shared memory from tile to tile is its own).  A release at cluster scope
// held the warp for 1-2.6k clocks per tile until its stores before were visible to the peer (18,944 x 3072 x 768 with
// GELU 108.2 us, relaxed 102.3).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load whose completion is counted on a barrier that may live in the peer CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tmap, uint32_t bar_cluster_addr,
                                                 int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
// Arrive on the barrier at this shared-memory offset in BOTH CTAs of the pair once every
// tcgen05 operation issued so far has retired.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
gemm_f16_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                     const __grid_constant__ CUtensorMap tm_out, const GemmArgs args) {
  using Cfg = PairCfg;
  constexpr int kStages = Cfg::kStages;
  constexpr int kTileN = Cfg::kTileN;
  constexpr bool kHasResidual = (EPI == BT_EPI_BIAS_RESIDUAL || EPI == BT_EPI_BIAS_RESIDUAL_F32OUT);

  // Both CTAs of the pair must use identical shared-memory offsets (the MMA and the multicast
  // commit address the peer by offset); dynamic shared memory starts at the same offset in
  // every CTA of a launch.
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const bool smem_ok = smem_aligned(args, smem_raw);
  uint8_t* smem = round_up_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes + Cfg::kStagingBytes);
  uint64_t* full_bar = bars;                    // [kStages]  (leader's copy is the live one)
  uint64_t* empty_bar = bars + kStages;         // [kStages]
  uint64_t* acc_full = bars + 2 * kStages;      // [2]
  uint64_t* acc_empty = bars + 2 * kStages + 2; // [2]        (leader's copy is the live one)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_int(static_cast<int>(threadIdx.x >> 5));  // warp-uniform roles: see common.cuh
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = uniform_u32(cluster_ctarank());  // 0 = leader
  const bool leader = cta_rank == 0;
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;

  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 2 * kEpiWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything is signalled across the pair
  tc_fence_after();
  const uint32_t tmem_base = uniform_u32(*tmem_slot);

  const int n_tiles = args.N / kTileN;
  const int num_kb = args.K / kBlockK;
  // The leading W blocks of the pair's first tile ahead of the dependency wait, its A blocks right behind it (see
  // gemm_f16_kernel).  Both CTAs' copies complete on the leader's barrier, which the leader arms for both.
  const int pre_kb = args.early_w && smem_ok ? (num_kb < kStages ? num_kb : kStages) : 0;
  auto load_w = [&](int stage, int n0, int kb) {
    uint8_t* sb = smem + stage * Cfg::kStageBytes + kABytes;
    const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
    if (elect_one()) tma_load_2d_pair(sb, &tm_b, bar, n0, kb * kBlockK);
    if (elect_one()) tma_load_2d_pair(sb + 64 * kBlockK * 2, &tm_b, bar, n0 + 64, kb * kBlockK);
  };
  auto load_a = [&](int stage, int m0, int kb) {
    const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
    if (elect_one()) tma_load_2d_pair(smem + stage * Cfg::kStageBytes, &tm_a, bar, kb * kBlockK, m0);
  };
  auto tile_rows = [&](int tile) { return (tile / n_tiles) * (2 * kBlockM) + static_cast<int>(cta_rank) * kBlockM; };
  auto tile_w_cols = [&](int tile) { return (tile % n_tiles) * kTileN + static_cast<int>(cta_rank) * 128; };
  if (warp == 0) {
    if (elect_one()) tma_prefetch_desc(&tm_a);
    if (elect_one()) tma_prefetch_desc(&tm_b);
    if (elect_one()) tma_prefetch_desc(&tm_out);
    for (int kb = 0; kb < pre_kb; ++kb) {
      if (leader && elect_one()) mbar_arrive_expect_tx(&full_bar[kb], 2 * Cfg::kStageBytes);
      load_w(kb, tile_w_cols(cluster_id), kb);
    }
  }

  pdl_wait();  // see gemm_f16_kernel
  if (warp == 0)
    for (int kb = 0; kb < pre_kb; ++kb) load_a(kb, tile_rows(cluster_id), kb);
  int M = args.m_rows;
  if (args.m_dev != nullptr) {
    const int md = __ldg(args.m_dev);
    M = uniform_int(md < M ? md : M);
  }
  if (!smem_ok) M = 0;
  const int m_tiles = (M + 2 * kBlockM - 1) / (2 * kBlockM);
  const int total_tiles = m_tiles * n_tiles;

  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    if (cluster_id >= total_tiles && leader) {
      // No tile for this pair after all: wait for the armed stages, so that no copy is in flight at exit.
      for (int kb = 0; kb < pre_kb; ++kb)
        if (!mbar_wait_warp(&full_bar[kb], 0u, abort_flag, args.status, kStatusGemmProducerTimeout)) break;
    }
    for (int tile = cluster_id; tile < total_tiles && ok; tile += num_clusters) {
      const int m0 = tile_rows(tile), n0 = tile_w_cols(tile);
      for (int kb = 0; kb < num_kb; ++kb) {
        if (tile != cluster_id || kb >= pre_kb) {  // else armed and requested above (stage == kb)
          if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1u, abort_flag, args.status, kStatusGemmProducerTimeout)) {
            ok = false;
            break;
          }
          // the leader announces the bytes of both CTAs; all copies complete on its barrier
          if (leader && elect_one()) mbar_arrive_expect_tx(&full_bar[stage], 2 * Cfg::kStageBytes);
          load_a(stage, m0, kb);
          load_w(stage, n0, kb);
        }
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------- MMA issuer (leader CTA only)
    if (leader) {
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true, landed = false;
      for (int tile = cluster_id; tile < total_tiles && ok; tile += num_clusters, ++it) {
        const int as = it & 1;
        const uint32_t aphase = (it >> 1) & 1;
        if (!mbar_wait_warp(&acc_empty[as], aphase ^ 1u, abort_flag, args.status, kStatusGemmMmaTimeout)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (lane == 0) gstamp(args.timing, it, 0);
        const uint32_t d_tmem = tmem_base + as * kTileN;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_latched(ok, landed, &full_bar[stage], phase, abort_flag, args.status, kStatusGemmMmaTimeout);
          tc_fence_after();
          const int cur = stage;
          const uint32_t sa = smem_u32(smem + cur * Cfg::kStageBytes);
          const uint32_t sb = sa + kABytes;
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
          landed = mbar_test_wait(&full_bar[stage], phase);  // the next block, ahead of these MMAs
          // (the commit frees the stage once these MMAs have retired)
          umma_k_block<true>(d_tmem, smem_desc(args.a_desc_hi, sa), smem_desc(args.b_desc_hi, sb), args.a_kstep_bytes >> 4,
                       args.b_kstep_bytes >> 4, args.idesc, kb != 0 ? 1u : 0u, &empty_bar[cur]);
        }
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (ok && elect_one()) umma_commit_pair(&acc_full[as]);
        if (lane == 0) gstamp(args.timing, it, 1);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int e = warp - 2;
    const int quarter = warp & 3;
    const int col_half = e >> 2;
    uint8_t* stg = smem + kStages * Cfg::kStageBytes + e * (Cfg::kStagingBufs * kStagingBytesPerWarp);
    __half* bias_s = bias_slice<kTileN>(bars, e);
    int it = 0;
    for (int tile = cluster_id; tile < total_tiles; tile += num_clusters, ++it) {
      const int m0 = (tile / n_tiles) * (2 * kBlockM) + static_cast<int>(cta_rank) * kBlockM;
      const int n0 = (tile % n_tiles) * kTileN;
      const int as = it & 1;
      const uint32_t aphase = (it >> 1) & 1;
      uint4 resv[kHasResidual ? kTileN / 16 : 1];
      prefetch_residual<kTileN, EPI>(args, m0, n0, M, quarter, col_half, lane, resv);
      BiasShare<kTileN> bias;
      if (EPI != BT_EPI_NONE) bias.load(args.bias, n0, col_half, lane);
      mbar_wait_anyway(&acc_full[as], aphase, abort_flag, args.status, kStatusGemmEpilogueTimeout);
      tc_fence_after();
      if (EPI != BT_EPI_NONE) bias.put(bias_s, lane);
      if (warp == 2 && lane == 0) gstamp(args.timing, it, 2);
      epilogue_tile<kTileN, EPI, true, Cfg::kStagingBufs>(args, &tm_out, stg, tmem_base + as * kTileN, m0, n0, M,
                                                          quarter, col_half, lane, resv,
                                                          reinterpret_cast<const uint4*>(bias_s));
      if (warp == 2 && lane == 0) gstamp(args.timing, it, 3);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[as]), 0));
    }
    if (lane == 0) tma_store_wait_all();
  }

  // ------------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  cluster_sync_all();  // neither CTA leaves while the other may still signal its barriers
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
  }
}

// ------------------------------------------------------------------------------------------
// GEMM + bias + residual + LayerNorm in one kernel:  y = LN(A*W + bias + residual)*gamma + beta.
// Main loop as in gemm_f16_kernel: tile t = (row tile t / C, column tile t % C), C = N / tile width, tiles round-robin over
// the CTAs, so the C column tiles of a row tile are worked on by C neighbouring CTAs at about the same time.  The
// pre-normalisation tensor never goes to HBM.  An epilogue warp owns 32 rows and 64 columns of the tile (16 warps for 256
// columns, 12 for 192, 8 for 128), a thread one row's 64 values, which stay in its registers from the first touch to the last (20 warps
// leave 96 registers a thread, which is why two warps of their own deal with the statistics):
//   1. v = accumulator + bias + residual, with the sum and sum of squares of v - s (s = the thread's first value: shifted
//      one-pass statistics).  The accumulator goes back to the MMA warp as soon as it has been read;
//   2. its (mean_i, M2_i) goes to shared memory, where one of two statistics warps merges the row's column groups;
//   3. that warp publishes the tile's (mean_i, M2_i) to a global scratch (it stays in L2) as two 64-bit
//      words, side by side with those of the slab's other rows, each (value bits << 32 | epoch of this launch): an aligned
//      64-bit store is single-copy atomic, so the tag validates the value and no fence or counter is needed.  It polls
//      (bounded) the 2*C words of the row until all carry the epoch, merges the C partials (equal counts n)
//         mean = avg(mean_i),  M2 = sum(M2_i) + n * sum((mean_i - mean)^2)
//      and hands mean and 1 / deviation to the row's threads;
//   4. normalise, gamma / beta, fp16, staging, TMA store.
// us per launch of 4,100 rows x 768 columns: with 128 values per thread (8 warps), written back to tensor memory for step 4,
// K = 768 / 3072 14.5 / 25.0; so 13.6 / 24.6 with 256 columns still and 12.4 / 20.7 with 192 (with the launch's memset).
// Accumulators are double buffered, so 1-4 of a tile overlap the main loop of the CTA's next
// tile.  A CTA only ever waits for the C CTAs working on the same row tile, and those wait for
// nothing but that row tile in turn, so the waits are never circular.  Progress does need those
// C neighbouring CTAs to be resident together: the grid never exceeds the SM count and a CTA
// takes a whole SM, so they are as soon as the kernels before have left; should something else hold
// SMs for long (another process, a hung kernel on another stream), the wait, bounded like every
// other wait of the library, gives up and reports kStatusGemmEpilogueTimeout instead of spinning.
// The scratch (16 * C bytes per row) must not hold this launch's epoch in the low half of any
// word beforehand: the caller zeroes it once and numbers the launches that share it 1, 2, 3, ...
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void st_relaxed_gpu_2u64(unsigned long long* p, unsigned long long v0, unsigned long long v1) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v0), "l"(v1) : "memory");
}
__device__ __forceinline__ void ld_relaxed_gpu_2u64(const unsigned long long* p, unsigned long long& v0,
                                                    unsigned long long& v1) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v0), "=l"(v1) : "l"(p) : "memory");
}
// Tile width of the one-CTA GEMM + LayerNorm kernel for this many row tiles on `ctas` CTAs: the width whose waves of tiles
// take least.  Clocks: a tile's main loop `k_block` per K block of 64, its epilogue `epilogue`; the epilogue of all waves
// but the last runs under the next wave's main loop, and a wave more costs 1.5k besides.  us per launch with its memset,
// widths 128 / 192 / 256 (64 columns were measured too: within 0.3 us of 128 at best).  768 columns, K = 768: 12 row tiles
// 10.9 / 11.4 / 12.7, 25 14.0 / 12.1 / 13.5, 38 14.7 / 15.6 / 13.8, 50 18.2 / 15.9 / 18.2; K = 3072: 12 17.3 / 19.6 /
// 23.2, 25 25.2 / 20.3 / 24.4, 38 25.8 / 32.3 / 24.9, 50 34.6 / 33.5 / 40.7, 74 41.9 / 39.8 / 49.4.  1024 columns (128 /
// 256), K = 1024: 16 12.1 / 14.5, 20 15.6 / 14.6, 38 20.7 / 21.5, 64 25.0 / 21.8.
struct LnWidthCost { int cols, k_block, epilogue; };
__host__ __device__ __forceinline__ int ln_tile_n(int m_tiles, int N, int K, int ctas) {
  constexpr LnWidthCost kCosts[3] = {{128, 290, 3700}, {192, 410, 4200}, {256, 520, 5600}};
  int best = 256;
  float best_cost = 3.0e38f;
  const float inv = 1.0f / static_cast<float>(ctas);
  const float blocks = static_cast<float>(K / kBlockK);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const LnWidthCost w = kCosts[i];
    if (N % w.cols != 0) continue;
    const float main = blocks * static_cast<float>(w.k_block), epi = static_cast<float>(w.epilogue);
    const float waves = ceilf(static_cast<float>(m_tiles * (N / w.cols)) * inv - 1.0e-4f);
    const float cost = main + epi + (waves - 1.0f) * (fmaxf(main, epi) + 1500.0f);
    if (cost <= best_cost) {  // (the wider of two that take the same)
      best_cost = cost;
      best = w.cols;
    }
  }
  return best;
}

constexpr int kLnEpiWarps = 16;
constexpr int kLnFirstEpiWarp = 4;      // warps 0 and 1 load and multiply, 2 and 3 exchange the statistics
constexpr int kLnThreads = 32 * (kLnFirstEpiWarp + kLnEpiWarps);
constexpr int kLnBarBytes = 384;          // barriers and slots
constexpr int kLnVecBytes = 256 * (4 + 4 + 2);  // gamma | beta | bias of a tile's columns: fp32, fp32, fp16

// Barriers between the epilogue warps and the two statistics warps.
struct LnBars {
  uint64_t* acc_full;   // [2]
  uint64_t* vec_full;   // bias / gamma / beta of the tile's columns are in shared memory
  uint64_t* vec_empty;  // all epilogue warps are done with them
  uint64_t* part;       // [4] all column groups' partials of a quarter's rows are in the staging buffers
  uint64_t* stat;       // [4] mean and 1 / deviation of a quarter's rows are there
  uint64_t* res;        // [kLnEpiWarps] a warp's residual rows have landed in its staging buffer
};
__device__ __forceinline__ LnBars ln_bars_at(uint64_t* acc_full) {
  return LnBars{acc_full, acc_full + 4, acc_full + 5, acc_full + 6, acc_full + 10, acc_full + 14};
}
template <int TILE_N>
__device__ __forceinline__ void init_ln_bars(const LnBars& b) {
  constexpr int kGroups = TILE_N / 64;
  mbar_init(b.vec_full, 1);
  mbar_init(b.vec_empty, 4 * kGroups);
  for (int q = 0; q < 4; ++q) {
    mbar_init(&b.part[q], kGroups);
    mbar_init(&b.stat[q], 1);
  }
  for (int w = 0; w < kLnEpiWarps; ++w) mbar_init(&b.res[w], 1);
}
// Where a row's partial and then its mean and 1 / deviation lie in a warp's staging buffer, between the reads of the
// residual and the writes of the output (a 16-byte unit that differs from row to row: four lanes to a bank).
__device__ __forceinline__ float2* ln_row_slot(uint8_t* stg, int lane) {
  return reinterpret_cast<float2*>(stg + lane * 128 + ((lane & 7) << 4));
}

// The epilogue warps' loop of the GEMM + LayerNorm kernels (one-CTA and pair form share it): steps 1, 2 and 4
// of the description above for every tile that `tile_at(it, m0, n0)` yields (m0 = first of this CTA's 128
// rows, n0 = first of the tile's columns); `release_acc(as)` hands accumulator buffer `as` back to the
// MMA issuer.  `stg_base`: a staging buffer of 4 KB per warp.
template <int TILE_N, class TileAt, class ReleaseAcc>
__device__ __forceinline__ void ln_epilogue_loop(const GemmArgs& args, const CUtensorMap* tm_out,
                                                 const CUtensorMap* tm_res, uint8_t* stg_base, const LnBars& bars,
                                                 const float* vec_s, volatile int* abort_flag, uint32_t tmem_base, int M,
                                                 int warp, int lane, TileAt tile_at, ReleaseAcc release_acc) {
  constexpr int kCols = 64;  // columns per thread
  const int e = warp - kLnFirstEpiWarp;
  const int quarter = warp & 3;
  const int cg = e >> 2;  // column group
  if (cg >= TILE_N / kCols) return;
  uint8_t* stg = stg_base + e * kStagingBytesPerWarp;
  uint8_t* srow = stg + lane * 128;
  int m0 = 0, n0 = 0;
  for (int it = 0; tile_at(it, m0, n0); ++it) {
    const int as = it & 1;
    const uint32_t aphase = (it >> 1) & 1;
    const int row0 = m0 + quarter * 32;
    const int gcol0 = n0 + cg * kCols;  // first of this thread's columns
    // Residual rows of this warp (32 rows x 64 columns) come through its staging buffer by TMA: row-strided 16-byte
    // loads from the threads would cost one L1 tag look-up per lane and load (4096 per tile), which alone took longer
    // than the main loop.
    if (lane == 0) {
      tma_store_wait_read_n<0>();  // the bulk store of the previous tile has read the buffer
      mbar_arrive_expect_tx(&bars.res[e], kStagingBytesPerWarp);
      tma_load_2d(stg, tm_res, &bars.res[e], gcol0, row0);
    }
    mbar_wait_anyway(&bars.acc_full[as], aphase, abort_flag, args.status, kStatusGemmEpilogueTimeout);
    tc_fence_after();
    if (e == 0 && lane == 0) gstamp(args.timing, it, 2);
    uint32_t v[64];
    const uint32_t t_row = tmem_base + as * TILE_N + (static_cast<uint32_t>(quarter * 32) << 16) + cg * kCols;
    tmem_ld_32x32_at<0>(t_row, v);
    tmem_ld_32x32_at<32>(t_row + 32, v);
    mbar_wait_anyway(bars.vec_full, it & 1u, abort_flag, args.status, kStatusGemmEpilogueTimeout);
    mbar_wait_anyway(&bars.res[e], it & 1u, abort_flag, args.status, kStatusGemmEpilogueTimeout);
    tmem_ld_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) release_acc(as);
    // ---- 1. v = acc + bias + residual; shifted sums
    const uint4* sbias = reinterpret_cast<const uint4*>(vec_s + 512) + cg * (kCols / 8);
    {
      float shift0 = 0.f;
      unsigned long long sd2 = pack_f32x2(0.f, 0.f), sdd2 = sd2, nshift2 = sd2;
#pragma unroll
      for (int q = 0; q < kCols / 8; ++q) {
        const uint4 r4 = *reinterpret_cast<const uint4*>(srow + ((q ^ (lane & 7)) << 4));
        const uint4 b4 = sbias[q];
        const uint32_t rh[4] = {r4.x, r4.y, r4.z, r4.w}, bh[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = q * 8 + 2 * j;
          float v0 = __uint_as_float(v[i]), v1 = __uint_as_float(v[i + 1]);
          add_half2(v0, v1, bh[j]);
          add_half2(v0, v1, rh[j]);
          if (i == 0) {
            shift0 = v0;
            nshift2 = pack_f32x2(-v0, -v0);
          }
          const unsigned long long d2 = add_f32x2(pack_f32x2(v0, v1), nshift2);
          sd2 = add_f32x2(sd2, d2);
          sdd2 = fma_f32x2(d2, d2, sdd2);
          v[i] = __float_as_uint(v0);
          v[i + 1] = __float_as_uint(v1);
        }
      }
      float s0, s1, q0, q1;
      unpack_f32x2(sd2, s0, s1);
      unpack_f32x2(sdd2, q0, q1);
      const float sd = s0 + s1, sdd = q0 + q1;
      // ---- 2. (the slot lies in residual columns that a lane reads itself, so no other lane waits for them)
      *ln_row_slot(stg, lane) =
          make_float2(shift0 + sd * (1.0f / kCols), fmaxf(sdd - sd * sd * (1.0f / kCols), 0.f));
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.part[quarter]);
    if (e == 0 && lane == 0) gstamp(args.timing, it, 4);
    mbar_wait_anyway(&bars.stat[quarter], it & 1u, abort_flag, args.status, kStatusGemmEpilogueTimeout);
    const float2 stat = *ln_row_slot(stg, lane);
    if (e == 0 && lane == 0) gstamp(args.timing, it, 6);
    const float shift = -stat.x * stat.y;
    const unsigned long long rstd2 = pack_f32x2(stat.y, stat.y), shift2 = pack_f32x2(shift, shift);
    // ---- 4. normalise, gamma / beta, fp16, store (64 columns = 128 B per row)
    const float4* sgamma = reinterpret_cast<const float4*>(vec_s + cg * kCols);
    const float4* sbeta = reinterpret_cast<const float4*>(vec_s + 256 + cg * kCols);
    const bool slab_full = row0 + 32 <= M;
#pragma unroll
    for (int q = 0; q < kCols / 8; ++q) {
      uint32_t u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = q * 8 + 2 * j;
        const float4 g4 = sgamma[2 * q + (j >> 1)], b4 = sbeta[2 * q + (j >> 1)];
        const unsigned long long n2 =
            fma_f32x2(pack_f32x2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), rstd2, shift2);
        float y0, y1;
        unpack_f32x2(fma_f32x2(n2, (j & 1) ? pack_f32x2(g4.z, g4.w) : pack_f32x2(g4.x, g4.y),
                               (j & 1) ? pack_f32x2(b4.z, b4.w) : pack_f32x2(b4.x, b4.y)), y0, y1);
        u[j] = pack_half2(y0, y1);
      }
      *reinterpret_cast<uint4*>(srow + ((q ^ (lane & 7)) << 4)) = make_uint4(u[0], u[1], u[2], u[3]);
    }
    if (!slab_full && row0 + lane < M) {  // (each lane its own row)
      __half* op = args.out_ln + static_cast<size_t>(row0 + lane) * args.N + gcol0;
#pragma unroll 1
      for (int q = 0; q < kCols / 8; ++q)
        reinterpret_cast<uint4*>(op)[q] = *reinterpret_cast<const uint4*>(srow + ((q ^ (lane & 7)) << 4));
    }
    // (the fence also puts this tile's accesses to the staging rows before the next tile's bulk write into them)
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (slab_full) {
        tma_store_2d(tm_out, stg, gcol0, row0);
        tma_store_commit();
      }
      mbar_arrive(bars.vec_empty);
    }
    if (e == 0 && lane == 0) gstamp(args.timing, it, 3);
  }
  if (lane == 0) tma_store_wait_all();
}

__device__ __forceinline__ void load8(float (&f)[8], const __half* p) {
  const uint4 h = __ldg(reinterpret_cast<const uint4*>(p));
  const __half2* hh = reinterpret_cast<const __half2*>(&h);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __half22float2(hh[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
__device__ __forceinline__ void load8(float (&f)[8], const float* p) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
  f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// The statistics warps' loop (`half` 0 or 1: quarters 2 * half and 2 * half + 1, a lane has one row of each): step 3.  The
// first of them also brings the tile's bias / gamma / beta slices into shared memory.
template <int TILE_N, class TileAt>
__device__ __forceinline__ void ln_statistics_loop(const GemmArgs& args, uint8_t* stg_base, const LnBars& bars, float* vec_s,
                                                   volatile int* abort_flag, int M, int n_tiles, int half, int lane,
                                                   TileAt tile_at) {
  constexpr int kGroups = TILE_N / 64;
  constexpr int kMaxParts = 1024 / TILE_N;  // column tiles of a row, N <= 1024
  const float inv_n = 1.0f / static_cast<float>(args.N);
  const float inv_tiles = 1.0f / static_cast<float>(n_tiles);
  const uint32_t epoch = args.ln_epoch;
  int m0 = 0, n0 = 0;
  for (int it = 0; tile_at(it, m0, n0); ++it) {
    if (half == 0) {
      float vec[2][8] = {};
      uint4 bias = make_uint4(0u, 0u, 0u, 0u);
      if (lane < TILE_N / 8) {
        const size_t at = n0 + lane * 8;
        bias = __ldg(reinterpret_cast<const uint4*>(args.bias + at));
        if (args.gb_fp32) {
          load8(vec[0], reinterpret_cast<const float*>(args.gamma) + at);
          load8(vec[1], reinterpret_cast<const float*>(args.beta) + at);
        } else {
          load8(vec[0], reinterpret_cast<const __half*>(args.gamma) + at);
          load8(vec[1], reinterpret_cast<const __half*>(args.beta) + at);
        }
      }
      mbar_wait_anyway(bars.vec_empty, (it & 1u) ^ 1u, abort_flag, args.status, kStatusGemmEpilogueTimeout);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        float4* dst = reinterpret_cast<float4*>(vec_s + k * 256 + lane * 8);
        dst[0] = make_float4(vec[k][0], vec[k][1], vec[k][2], vec[k][3]);
        dst[1] = make_float4(vec[k][4], vec[k][5], vec[k][6], vec[k][7]);
      }
      reinterpret_cast<uint4*>(vec_s + 512)[lane] = bias;
      __syncwarp();
      if (lane == 0) mbar_arrive(bars.vec_full);
    }
    // The words of a partial's 32 rows lie side by side, so that a warp writes or reads them with one
    // instruction on four whole lines (the allocation's last slab may have fewer than 32 rows).
    unsigned long long* words[2];
    int slab_rows[2];
    bool row_ok[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int quarter = 2 * half + k;
      const int row0 = m0 + quarter * 32;
      slab_rows[k] = min(32, args.m_rows - row0);
      words[k] = reinterpret_cast<unsigned long long*>(args.out) + static_cast<size_t>(row0) * n_tiles * 2;
      row_ok[k] = row0 + lane < M;
      mbar_wait_anyway(&bars.part[quarter], it & 1u, abort_flag, args.status, kStatusGemmEpilogueTimeout);
      float gm[kGroups], gq[kGroups], mean = 0.f, m2 = 0.f;
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        // (quarter q is that of the warps 4 g + q from kLnFirstEpiWarp, a multiple of four, on)
        const float2 f = *ln_row_slot(stg_base + (g * 4 + quarter) * kStagingBytesPerWarp, lane);
        gm[g] = f.x;
        gq[g] = f.y;
        mean += f.x;
      }
      mean *= 1.0f / kGroups;
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const float d = gm[g] - mean;
        m2 += gq[g] + 64.0f * d * d;
      }
      // A naturally aligned 64-bit store is single-copy atomic, so a reader that finds this launch's epoch in a word
      // also has its value: no fence, no counter, no second round trip.
      if (row_ok[k])
        st_relaxed_gpu_2u64(words[k] + ((n0 / TILE_N) * slab_rows[k] + lane) * 2,
                            (static_cast<unsigned long long>(__float_as_uint(mean)) << 32) | epoch,
                            (static_cast<unsigned long long>(__float_as_uint(m2)) << 32) | epoch);
    }
    if (half == 0 && lane == 0) gstamp(args.timing, it, 5);
    // Wait until the rows' 2 * n_tiles words all carry this epoch (bounded), then merge.
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int quarter = 2 * half + k;
      float pm[kMaxParts], pq[kMaxParts];
      const long long t0 = clock64();
      uint32_t probes = 0;
      while (true) {
        uint32_t bad = 0;
        if (row_ok[k]) {
          // all loads are issued before any tag is looked at: one round trip
#pragma unroll
          for (int p = 0; p < kMaxParts; ++p)
            if (p < n_tiles) {
              unsigned long long w0, w1;
              ld_relaxed_gpu_2u64(words[k] + (p * slab_rows[k] + lane) * 2, w0, w1);
              bad |= (static_cast<uint32_t>(w0) ^ epoch) | (static_cast<uint32_t>(w1) ^ epoch);
              pm[p] = __uint_as_float(static_cast<uint32_t>(w0 >> 32));
              pq[p] = __uint_as_float(static_cast<uint32_t>(w1 >> 32));
            }
        }
        if (__all_sync(0xffffffffu, bad == 0)) break;
        if ((++probes & 15u) == 0u && __any_sync(0xffffffffu, *abort_flag != 0 || clock64() - t0 > (1ll << 31))) {
          if (lane == 0) {
            *abort_flag = 1;
            if (args.status != nullptr) atomicCAS(args.status, 0, kStatusGemmEpilogueTimeout);
          }
          break;
        }
      }
      float mean = 0.f, rstd = 0.f;
      if (row_ok[k]) {
#pragma unroll
        for (int p = 0; p < kMaxParts; ++p)
          if (p < n_tiles) mean += pm[p];
        mean *= inv_tiles;
        float M2 = 0.f;
#pragma unroll
        for (int p = 0; p < kMaxParts; ++p)
          if (p < n_tiles) {
            const float d = pm[p] - mean;
            M2 += pq[p] + static_cast<float>(TILE_N) * d * d;
          }
        rstd = rsqrtf(M2 * inv_n + args.eps);
      }
#pragma unroll
      for (int g = 0; g < kGroups; ++g)
        *ln_row_slot(stg_base + (g * 4 + quarter) * kStagingBytesPerWarp, lane) = make_float2(mean, rstd);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.stat[quarter]);
    }
  }
}

// The rows that are there; none where shared memory is not aligned.
__device__ __forceinline__ int ln_rows(const GemmArgs& args, const uint8_t* smem) {
  int M = args.m_rows;
  if (args.m_dev != nullptr) {
    const int md = __ldg(args.m_dev);
    M = md < M ? md : M;
  }
  return uniform_int(smem_aligned(args, smem) ? M : 0);
}

template <int TILE_N>
struct LnCfg {
  static constexpr int kStageBytes = kABytes + TILE_N * kBlockK * 2;
  static constexpr int kStages = TILE_N == 256 ? 3 : TILE_N == 192 ? 4 : 6;
  static constexpr int kStagingBytes = (TILE_N / 64) * 4 * kStagingBytesPerWarp;
  static constexpr int kRingAndStaging = kStages * kStageBytes + kStagingBytes;
};
constexpr int kLnRingAndStaging = LnCfg<128>::kRingAndStaging;  // the largest of the three
static_assert(LnCfg<192>::kRingAndStaging <= kLnRingAndStaging && LnCfg<256>::kRingAndStaging <= kLnRingAndStaging, "");

// One width of gemm_f16_ln_kernel, from the barriers on.  `M` valid rows.  Warp 1 is told whether it has freed tensor memory.
template <int TILE_N>
__device__ __forceinline__ bool ln_gemm_body(const CUtensorMap* tm_a, const CUtensorMap* tm_b, const CUtensorMap* tm_out,
                                             const CUtensorMap* tm_res, const GemmArgs& args, uint8_t* smem,
                                             uint64_t* bars, float* vec_s, uint32_t* tmem_slot,
                                             volatile int* abort_flag, int M, int warp, int lane) {
  using Cfg = LnCfg<TILE_N>;
  constexpr int kStages = Cfg::kStages;
  uint64_t* full_bar = bars;                    // [kStages]
  uint64_t* empty_bar = bars + kStages;         // [kStages]
  uint64_t* acc_full = bars + 2 * kStages;      // [2]
  uint64_t* acc_empty = bars + 2 * kStages + 2; // [2]
  const LnBars ln_bars = ln_bars_at(acc_full);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 4 * (TILE_N / 64));
    }
    init_ln_bars<TILE_N>(ln_bars);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform_u32(*tmem_slot);

  const int n_tiles = args.N / TILE_N;
  const int num_kb = args.K / kBlockK;
  const int m_tiles = (M + kBlockM - 1) / kBlockM;
  const int total_tiles = m_tiles * n_tiles;
  auto tile_at = [&](int li, int& m0, int& n0) -> bool {
    const int tile = static_cast<int>(blockIdx.x) + li * static_cast<int>(gridDim.x);
    if (tile >= total_tiles) return false;
    m0 = (tile / n_tiles) * kBlockM;
    n0 = (tile % n_tiles) * TILE_N;
    return true;
  };
  // The leading W blocks of the first tile ahead of the dependency wait, its A blocks right behind it (see
  // gemm_f16_kernel).
  auto load_w = [&](int stage, int n0, int kb) {
    uint8_t* sb = smem + stage * Cfg::kStageBytes + kABytes;
#pragma unroll
    for (int c = 0; c < TILE_N / 64; ++c)
      if (elect_one()) tma_load_2d(sb + c * (64 * kBlockK * 2), tm_b, &full_bar[stage], n0 + c * 64, kb * kBlockK);
  };
  auto load_a = [&](int stage, int m0, int kb) {
    if (elect_one()) tma_load_2d(smem + stage * Cfg::kStageBytes, tm_a, &full_bar[stage], kb * kBlockK, m0);
  };
  int pre_kb = 0;
  if (warp == 0) {
    int m0 = 0, n0 = 0;
    if (tile_at(0, m0, n0)) {
      if (args.early_w) pre_kb = num_kb < kStages ? num_kb : kStages;
      for (int kb = 0; kb < pre_kb; ++kb) {
        if (elect_one()) mbar_arrive_expect_tx(&full_bar[kb], Cfg::kStageBytes);
        load_w(kb, n0, kb);
      }
    }
  }

  pdl_wait();  // see gemm_f16_kernel
  bool tmem_freed = false;

  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int m0 = 0, n0 = 0;
    for (int li = 0; ok && tile_at(li, m0, n0); ++li) {
      for (int kb = 0; kb < num_kb; ++kb) {
        if (li == 0 && kb < pre_kb) {  // armed above, its W block requested (stage == kb)
          load_a(stage, m0, kb);
        } else {
          if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1u, abort_flag, args.status, kStatusGemmProducerTimeout)) {
            ok = false;
            break;
          }
          if (elect_one()) mbar_arrive_expect_tx(&full_bar[stage], Cfg::kStageBytes);
          load_a(stage, m0, kb);
          load_w(stage, n0, kb);
        }
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // --------------------------------------------------------------- MMA issuer
    {
      constexpr uint32_t kIdesc = make_idesc_f16(kBlockM, TILE_N, 0, 1);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true, landed = false;
      int m0 = 0, n0 = 0, tiles = 0;
      for (int it = 0; ok && tile_at(it, m0, n0); ++it) {
        const int as = it & 1;
        const uint32_t aphase = (it >> 1) & 1;
        if (!mbar_wait_warp(&acc_empty[as], aphase ^ 1u, abort_flag, args.status, kStatusGemmMmaTimeout)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (lane == 0) gstamp(args.timing, it, 0);
        const uint32_t d_tmem = tmem_base + as * TILE_N;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_latched(ok, landed, &full_bar[stage], phase, abort_flag, args.status, kStatusGemmMmaTimeout);
          tc_fence_after();
          const int cur = stage;
          const uint32_t sa = smem_u32(smem + cur * Cfg::kStageBytes);
          const uint32_t sb = sa + kABytes;
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
          landed = mbar_test_wait(&full_bar[stage], phase);  // the next block, ahead of these MMAs
          // (the commit frees the stage once these MMAs have retired)
          umma_k_block<false>(d_tmem, smem_desc(args.a_desc_hi, sa), smem_desc(args.b_desc_hi, sb), args.a_kstep_bytes >> 4,
                       args.b_kstep_bytes >> 4, kIdesc, kb != 0 ? 1u : 0u, &empty_bar[cur]);
        }
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (ok && elect_one()) umma_commit(&acc_full[as]);
        if (lane == 0) gstamp(args.timing, it, 1);
        tiles = it + 1;
      }
      if (accumulators_back(acc_empty, tiles, abort_flag, args.status, kStatusGemmMmaTimeout)) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
        tmem_freed = true;
      }
    }
  } else if (warp < kLnFirstEpiWarp) {
    // ------------------------------------------------------- row statistics
    ln_statistics_loop<TILE_N>(args, smem + kStages * Cfg::kStageBytes, ln_bars, vec_s, abort_flag, M, n_tiles, warp - 2,
                               lane, tile_at);
  } else {
    // ------------------------------------------------------------------ epilogue
    ln_epilogue_loop<TILE_N>(args, tm_out, tm_res, smem + kStages * Cfg::kStageBytes, ln_bars, vec_s, abort_flag,
                             tmem_base, M, warp, lane, tile_at, [&](int as) { mbar_arrive(&acc_empty[as]); });
  }
  return tmem_freed;
}

__global__ void __launch_bounds__(kLnThreads, 1)
gemm_f16_ln_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                   const __grid_constant__ CUtensorMap tm_out, const __grid_constant__ CUtensorMap tm_res,
                   const GemmArgs args) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kLnRingAndStaging);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kLnRingAndStaging + kLnBarBytes - 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* vec_s = reinterpret_cast<float*>(smem + kLnRingAndStaging + kLnBarBytes);

  const int warp = uniform_int(static_cast<int>(threadIdx.x >> 5));  // warp-uniform roles: see common.cuh
  const int lane = threadIdx.x & 31;

  pdl_launch_dependents();

  // The row count is known ahead of the dependency wait (see common.cuh: inside a call this is never the second
  // kernel), so the tile width can go by the rows that are there instead of those that are allocated.
  const int M = ln_rows(args, smem);
  if (threadIdx.x == 0) *abort_flag = 0;
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
    tma_prefetch_desc(&tm_out);
    tma_prefetch_desc(&tm_res);
  }
  const int m_tiles = (M + kBlockM - 1) / kBlockM;
  const int tile_n = args.force_n != 0 ? args.force_n : ln_tile_n(m_tiles, args.N, args.K, static_cast<int>(gridDim.x));
  bool tmem_freed = false;
  if (tile_n == 128)
    tmem_freed = ln_gemm_body<128>(&tm_a, &tm_b, &tm_out, &tm_res, args, smem, bars, vec_s, tmem_slot, abort_flag, M, warp, lane);
  else if (tile_n == 192)
    tmem_freed = ln_gemm_body<192>(&tm_a, &tm_b, &tm_out, &tm_res, args, smem, bars, vec_s, tmem_slot, abort_flag, M, warp, lane);
  else
    tmem_freed = ln_gemm_body<256>(&tm_a, &tm_b, &tm_out, &tm_res, args, smem, bars, vec_s, tmem_slot, abort_flag, M, warp, lane);

  // ------------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    if (warp == 1 && !tmem_freed) {
      tc_fence_after();
      tmem_dealloc(*tmem_slot, 512);
    }
  }
}

// ------------------------------------------------------------------------------------------
// GEMM + bias + residual + LayerNorm on SM pairs: the main loop of gemm_f16_pair_kernel (256 x 256
// tiles, cta_group::2, half of the W tile per SM) with the epilogue of gemm_f16_ln_kernel.  Each CTA
// of a pair holds the accumulator of its own 128 rows, so its epilogue warps do exactly what those of
// the one-CTA kernel do; the partials of a row come from the N/256 clusters working on that row tile.
// Tiles go round-robin over the clusters (all resident: the launch asks for no more clusters than fit),
// and a cluster only waits for clusters working on earlier or the same row tiles: no circular wait.
// ------------------------------------------------------------------------------------------
struct PairLnCfg {
  static constexpr int kTileN = 256;
  static constexpr int kStageBytes = PairCfg::kStageBytes;
  static constexpr int kStages = 5;  // (what 16 staging buffers leave room for)
  static constexpr int kTmemCols = 512;
  static constexpr int kStagingBytes = kLnEpiWarps * kStagingBytesPerWarp;
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kLnThreads, 1)
gemm_f16_pair_ln_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                        const __grid_constant__ CUtensorMap tm_out, const __grid_constant__ CUtensorMap tm_res,
                        const GemmArgs args) {
  using Cfg = PairLnCfg;
  constexpr int kStages = Cfg::kStages;
  constexpr int kTileN = Cfg::kTileN;

  // (both CTAs of a pair use the same shared-memory offsets: the MMA and the multicast commit address the peer by offset)
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes + Cfg::kStagingBytes);
  uint64_t* full_bar = bars;                    // [kStages]  (leader's copy is the live one)
  uint64_t* empty_bar = bars + kStages;         // [kStages]
  uint64_t* acc_full = bars + 2 * kStages;      // [2]
  uint64_t* acc_empty = bars + 2 * kStages + 2; // [2]        (leader's copy is the live one)
  const LnBars ln_bars = ln_bars_at(acc_full);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(bars) + kLnBarBytes - 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* vec_s = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + kLnBarBytes);

  const int warp = uniform_int(static_cast<int>(threadIdx.x >> 5));  // warp-uniform roles: see common.cuh
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = uniform_u32(cluster_ctarank());  // 0 = leader
  const bool leader = cta_rank == 0;
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;

  pdl_launch_dependents();

  const int M = ln_rows(args, smem);  // (ahead of the dependency wait, as in gemm_f16_ln_kernel)

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 2 * kLnEpiWarps);
    }
    init_ln_bars<kTileN>(ln_bars);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything is signalled across the pair
  tc_fence_after();
  const uint32_t tmem_base = uniform_u32(*tmem_slot);

  const int n_tiles = args.N / kTileN;
  const int num_kb = args.K / kBlockK;
  const int m_tiles = (M + 2 * kBlockM - 1) / (2 * kBlockM);
  const int total_tiles = m_tiles * n_tiles;
  // The leading W blocks of the pair's first tile ahead of the dependency wait, its A blocks right behind it (see
  // gemm_f16_kernel).  Both CTAs' copies complete on the leader's barrier, which the leader arms for both.
  const int pre_kb = args.early_w && cluster_id < total_tiles ? (num_kb < kStages ? num_kb : kStages) : 0;
  auto load_w = [&](int stage, int n0, int kb) {
    uint8_t* sb = smem + stage * Cfg::kStageBytes + kABytes;
    const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
    if (elect_one()) tma_load_2d_pair(sb, &tm_b, bar, n0, kb * kBlockK);
    if (elect_one()) tma_load_2d_pair(sb + 64 * kBlockK * 2, &tm_b, bar, n0 + 64, kb * kBlockK);
  };
  auto load_a = [&](int stage, int m0, int kb) {
    const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
    if (elect_one()) tma_load_2d_pair(smem + stage * Cfg::kStageBytes, &tm_a, bar, kb * kBlockK, m0);
  };
  auto tile_rows = [&](int tile) { return (tile / n_tiles) * (2 * kBlockM) + static_cast<int>(cta_rank) * kBlockM; };
  auto tile_w_cols = [&](int tile) { return (tile % n_tiles) * kTileN + static_cast<int>(cta_rank) * 128; };
  if (warp == 0) {
    if (elect_one()) tma_prefetch_desc(&tm_a);
    if (elect_one()) tma_prefetch_desc(&tm_b);
    if (elect_one()) tma_prefetch_desc(&tm_out);
    if (elect_one()) tma_prefetch_desc(&tm_res);
    for (int kb = 0; kb < pre_kb; ++kb) {
      if (leader && elect_one()) mbar_arrive_expect_tx(&full_bar[kb], 2 * Cfg::kStageBytes);
      load_w(kb, tile_w_cols(cluster_id), kb);
    }
  }

  pdl_wait();  // see gemm_f16_kernel
  if (warp == 0)
    for (int kb = 0; kb < pre_kb; ++kb) load_a(kb, tile_rows(cluster_id), kb);
  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = cluster_id; tile < total_tiles && ok; tile += num_clusters) {
      const int m0 = tile_rows(tile), n0 = tile_w_cols(tile);
      for (int kb = 0; kb < num_kb; ++kb) {
        if (tile != cluster_id || kb >= pre_kb) {  // else armed and requested above (stage == kb)
          if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1u, abort_flag, args.status, kStatusGemmProducerTimeout)) {
            ok = false;
            break;
          }
          // the leader announces the bytes of both CTAs; all copies complete on its barrier
          if (leader && elect_one()) mbar_arrive_expect_tx(&full_bar[stage], 2 * Cfg::kStageBytes);
          load_a(stage, m0, kb);
          load_w(stage, n0, kb);
        }
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------- MMA issuer (leader CTA only)
    if (leader) {
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true, landed = false;
      for (int tile = cluster_id; tile < total_tiles && ok; tile += num_clusters, ++it) {
        const int as = it & 1;
        const uint32_t aphase = (it >> 1) & 1;
        if (!mbar_wait_warp(&acc_empty[as], aphase ^ 1u, abort_flag, args.status, kStatusGemmMmaTimeout)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (lane == 0) gstamp(args.timing, it, 0);
        const uint32_t d_tmem = tmem_base + as * kTileN;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_latched(ok, landed, &full_bar[stage], phase, abort_flag, args.status, kStatusGemmMmaTimeout);
          tc_fence_after();
          const int cur = stage;
          const uint32_t sa = smem_u32(smem + cur * Cfg::kStageBytes);
          const uint32_t sb = sa + kABytes;
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
          landed = mbar_test_wait(&full_bar[stage], phase);  // the next block, ahead of these MMAs
          // (the commit frees the stage once these MMAs have retired)
          umma_k_block<true>(d_tmem, smem_desc(args.a_desc_hi, sa), smem_desc(args.b_desc_hi, sb), args.a_kstep_bytes >> 4,
                       args.b_kstep_bytes >> 4, args.idesc, kb != 0 ? 1u : 0u, &empty_bar[cur]);
        }
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (ok && elect_one()) umma_commit_pair(&acc_full[as]);
        if (lane == 0) gstamp(args.timing, it, 1);
      }
    }
  } else {
    // --------------------------------------------- epilogue and row statistics
    auto tile_at = [&](int it, int& m0, int& n0) -> bool {
      const int tile = cluster_id + it * num_clusters;
      if (tile >= total_tiles) return false;
      m0 = (tile / n_tiles) * (2 * kBlockM) + static_cast<int>(cta_rank) * kBlockM;
      n0 = (tile % n_tiles) * kTileN;
      return true;
    };
    if (warp < kLnFirstEpiWarp)
      ln_statistics_loop<kTileN>(args, smem + kStages * Cfg::kStageBytes, ln_bars, vec_s, abort_flag, M, n_tiles, warp - 2,
                                 lane, tile_at);
    else
      ln_epilogue_loop<kTileN>(args, &tm_out, &tm_res, smem + kStages * Cfg::kStageBytes, ln_bars, vec_s, abort_flag,
                               tmem_base, M, warp, lane, tile_at,
                               [&](int as) { mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[as]), 0)); });
  }

  // ------------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  cluster_sync_all();  // neither CTA leaves while the other may still signal its barriers
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
  }
}


// ------------------------------------------------------------------------------------------ launch
template <int BLOCK_N, int EPI>
cudaError_t launch_one(const GemmLaunch& g, const GemmArgs& a, cudaStream_t stream) {
  using Cfg = GemmCfg<BLOCK_N>;
  static bool attr_set[64] = {};  // per template instance and device
  auto kern = gemm_f16_kernel<BLOCK_N, EPI>;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  const int n_tiles = g.N / BLOCK_N;
  const int m_tiles = (g.m_rows + kBlockM - 1) / kBlockM;
  long long tiles = static_cast<long long>(n_tiles) * m_tiles * (EPI == kEpiSplitKF32 ? a.split_k : 1);
  int grid = static_cast<int>(tiles < g.num_sms ? tiles : g.num_sms);
  if (grid < 1) grid = 1;
  return launch_pdl(kern, dim3(grid), dim3(kGemmThreads), Cfg::kSmemBytes, stream, g.tm_a, g.tm_b, g.tm_out, a);
}

template <int BLOCK_N>
cudaError_t launch_epi(const GemmLaunch& g, const GemmArgs& a, cudaStream_t stream) {
  switch (g.epilogue) {
    case BT_EPI_NONE: return launch_one<BLOCK_N, BT_EPI_NONE>(g, a, stream);
    case BT_EPI_BIAS: return launch_one<BLOCK_N, BT_EPI_BIAS>(g, a, stream);
    case BT_EPI_BIAS_GELU:
      return g.gelu_kind == BT_GELU_TANH ? launch_one<BLOCK_N, kEpiBiasGeluTanh>(g, a, stream)
                                         : launch_one<BLOCK_N, BT_EPI_BIAS_GELU>(g, a, stream);
    case BT_EPI_BIAS_RESIDUAL: return launch_one<BLOCK_N, BT_EPI_BIAS_RESIDUAL>(g, a, stream);
    case BT_EPI_BIAS_RESIDUAL_F32OUT: return launch_one<BLOCK_N, BT_EPI_BIAS_RESIDUAL_F32OUT>(g, a, stream);
    default: return cudaErrorInvalidValue;
  }
}

// Clusters of two that can be co-resident on a device (one CTA per SM); 0 = not yet asked.
int g_pair_clusters[64] = {};

template <int EPI>
cudaError_t launch_pair(const GemmLaunch& g, const GemmArgs& a, cudaStream_t stream) {
  using Cfg = PairCfg;
  static bool attr_set[64] = {};
  auto kern = gemm_f16_pair_kernel<EPI>;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  if (g_pair_clusters[dev] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (g.num_sms / 2));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = g.num_sms / 2;
    }
    g_pair_clusters[dev] = n;
  }
  const int n_tiles = g.N / Cfg::kTileN;
  const int m_tiles = (g.m_rows + 2 * kBlockM - 1) / (2 * kBlockM);
  long long tiles = static_cast<long long>(n_tiles) * m_tiles;
  int clusters = static_cast<int>(tiles < g_pair_clusters[dev] ? tiles : g_pair_clusters[dev]);
  if (clusters < 1) clusters = 1;
  return launch_pdl(kern, dim3(2 * clusters), dim3(kGemmThreads), Cfg::kSmemBytes, stream, g.tm_a, g.tm_b, g.tm_out, a);
}

cudaError_t launch_pair_epi(const GemmLaunch& g, const GemmArgs& a, cudaStream_t stream) {
  switch (g.epilogue) {
    case BT_EPI_NONE: return launch_pair<BT_EPI_NONE>(g, a, stream);
    case BT_EPI_BIAS: return launch_pair<BT_EPI_BIAS>(g, a, stream);
    case BT_EPI_BIAS_GELU:
      return g.gelu_kind == BT_GELU_TANH ? launch_pair<kEpiBiasGeluTanh>(g, a, stream)
                                         : launch_pair<BT_EPI_BIAS_GELU>(g, a, stream);
    case BT_EPI_BIAS_RESIDUAL: return launch_pair<BT_EPI_BIAS_RESIDUAL>(g, a, stream);
    case BT_EPI_BIAS_RESIDUAL_F32OUT: return launch_pair<BT_EPI_BIAS_RESIDUAL_F32OUT>(g, a, stream);
    default: return cudaErrorInvalidValue;
  }
}

struct LnGemmCfg {
  static constexpr int kSmemBytes = kLnRingAndStaging + kLnBarBytes + kLnVecBytes;
};
static_assert(LnGemmCfg::kSmemBytes <= 227 * 1024, "shared memory of the GEMM + LayerNorm kernel");

struct PairLnGemmCfg {
  static constexpr int kSmemBytes = PairLnCfg::kStages * PairLnCfg::kStageBytes + PairLnCfg::kStagingBytes + kLnBarBytes + kLnVecBytes;
};
static_assert(PairLnGemmCfg::kSmemBytes <= 227 * 1024, "shared memory of the pair GEMM + LayerNorm kernel");
int g_pair_ln_clusters[64] = {};

// The pair form of the GEMM + LayerNorm kernel.  `a.idesc` must describe M = 256.
cudaError_t launch_pair_ln_gemm(const GemmLaunch& g, const GemmArgs& a, cudaStream_t stream) {
  using Cfg = PairLnGemmCfg;
  static bool attr_set[64] = {};
  auto kern = gemm_f16_pair_ln_kernel;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  if (g_pair_ln_clusters[dev] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (g.num_sms / 2));
    cfg.blockDim = dim3(kLnThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    int n = 0;
    // every cluster must be resident (clusters wait for one another's row statistics): without an
    // answer from the occupancy query the pair form is not used
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = -1;
    }
    g_pair_ln_clusters[dev] = n;
  }
  if (g_pair_ln_clusters[dev] <= 0) return cudaErrorNotSupported;
  const int n_tiles = g.N / 256;
  const int m_tiles = (g.m_rows + 2 * kBlockM - 1) / (2 * kBlockM);
  long long tiles = static_cast<long long>(n_tiles) * m_tiles;
  int clusters = static_cast<int>(tiles < g_pair_ln_clusters[dev] ? tiles : g_pair_ln_clusters[dev]);
  if (clusters < 1) clusters = 1;
  return launch_pdl(kern, dim3(2 * clusters), dim3(kLnThreads), Cfg::kSmemBytes, stream, g.tm_a, g.tm_b, g.tm_out,
                    g.tm_res, a);
}

// The pair form of GEMM + LayerNorm (main loop on SM pairs, half of the W tile per SM) is the faster one where there are
// waves enough that its coarser tiles fill them; below, the one-CTA form fits its width to the rows.  us per launch with
// its memset, one-CTA / pair form: 768 columns, K = 3072: 9,400 rows (two waves of 192-column tiles) 39.6 / 43.5, 12,500
// 54.6 / 51.2, 75,776 300 / 269; K = 768: 18,944 rows (four waves) 28.9 / 30.2, 28,000 41.2 / 40.3, 75,776 101 / 98.  1024
// columns (no 192; one wave is up to 4,736 rows), K = 4096: 4,100 rows 38.9 / 41.0, 6,200 74.5 / 60.3; K = 1024: 4,100 rows
// 22.7 / 24.5, 6,400 32.6 / 32.4, 12,500 38.4 / 36.0.  512 columns, K = 2048: 9,400 rows 22.3 / 23.3, 12,500 34.5 / 31.9.
// With a single column tile (256 columns) a long K is what counts, from more than one tile per SM pair on: K = 4096, 11,000
// rows 38.1 / 32.3, 18,944 46.1 / 40.2; K = 3072 28.8 / 25.5 and 37.6 / 34.0; K = 2048 19.9 / 20.6 and 25.0 / 22.6; 9,400
// rows, one wave of 128-column tiles, K = 3072 17.4 / 25.2.
bool ln_pair_pays(int m_rows, int N, int K, int num_sms) {
  const long long m_tiles = (m_rows + kBlockM - 1) / kBlockM;
  if (N % 192 == 0) return m_tiles * (N / 192) > (K >= 2048 ? 2LL : 4LL) * num_sms;
  if (N == 256 && K >= 2048) return 2 * m_tiles > num_sms;
  return m_tiles * (N / 256) > num_sms;
}

cudaError_t launch_ln_gemm(const GemmLaunch& g, const GemmArgs& a_in, cudaStream_t stream) {
  using Cfg = LnGemmCfg;
  static bool attr_set[64] = {};
  auto kern = gemm_f16_ln_kernel;
  if (g.N % 256 != 0 || g.N > 1024 || !g.out_ln || !g.gamma || !g.beta || !g.residual || !g.bias || g.ln_epoch == 0)
    return cudaErrorInvalidValue;
  const bool want_pair = g_dbg_ln_pair == 1 || (g_dbg_ln_pair == 0 && ln_pair_pays(g.m_rows, g.N, g.K, g.num_sms));
  if (want_pair) {
    GemmArgs ap = a_in;
    ap.idesc = make_idesc_f16(256, 256, 0, 1);
    const cudaError_t e = launch_pair_ln_gemm(g, ap, stream);
    if (e != cudaErrorNotSupported) return e;
  }
  const GemmArgs& a = a_in;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  const int m_tiles = (g.m_rows + kBlockM - 1) / kBlockM;
  const long long tiles = static_cast<long long>(m_tiles) * (g.N / 128);  // the narrowest width's
  int grid = static_cast<int>(tiles < g.num_sms ? tiles : g.num_sms);
  if (grid < 1) grid = 1;
  return launch_pdl(kern, dim3(grid), dim3(kLnThreads), Cfg::kSmemBytes, stream, g.tm_a, g.tm_b, g.tm_out, g.tm_res, a);
}

// The pair kernel needs N % 256 == 0 and pays off once every SM pair gets at least two
// 256 x 256 tiles (below that the narrower one-CTA tiles fill the machine better).
bool use_pair_kernel(const GemmLaunch& g) {
  if (g.epilogue == BT_EPI_BIAS_RESIDUAL_LAYERNORM) return false;
  if (g_dbg_pair_mode == 1) return g.N % 256 == 0;
  if (g_dbg_pair_mode == 2 || g_dbg_force_block_n != 0 || g.block_n != 0) return false;
  if (g.N % 256 != 0) return false;
  // Measured at 18.9k rows: with a short main loop (K = 768) the fp32 + residual epilogue bounds
  // the tile time and the one-CTA kernel is a few percent faster.  (The GELU epilogue used to be
  // on that list; with the present epilogue the pair kernel gains 1.6 % on the whole forward.)
  if ((g.epilogue == BT_EPI_BIAS_RESIDUAL || g.epilogue == BT_EPI_BIAS_RESIDUAL_F32OUT) && g.K < 2048) return false;
  const long long tiles = static_cast<long long>((g.m_rows + 255) / 256) * (g.N / 256);
  return tiles >= 2LL * (g.num_sms / 2);
}

}  // namespace

// Few rows and a long K leave most SMs idle while a handful stream the weights one K block
// after the other; cutting K spreads that stream.  The widest cut whose (tile, range) pairs number at
// most one and a half times the SMs (the row count is an upper bound: padded rows make no tiles), with
// at least three K blocks per range.
int gemm_pick_split_k(int m_rows, int N, int K, int num_sms) {
  if (N % 64 != 0 || K % kBlockK != 0) return 1;
  if (g_dbg_split_k != 0)
    return (g_dbg_split_k > 0 && (K / kBlockK) % g_dbg_split_k == 0) ? static_cast<int>(g_dbg_split_k) : 1;
  const long long tiles = static_cast<long long>((m_rows + kBlockM - 1) / kBlockM) * (N / 64);
  const int num_kb = K / kBlockK;
  const int cands[3] = {8, 4, 2};
  for (int i = 0; i < 3; ++i) {
    const int s = cands[i];
    if (num_kb % s != 0 || num_kb / s < 3) continue;
    if (tiles * s <= num_sms + num_sms / 2) return s;
  }
  return 1;
}

int gemm_pick_block_n(int m_rows, int N, int K, int num_sms, bool all_rows) {
  if (g_dbg_force_block_n != 0) return static_cast<int>(g_dbg_force_block_n);
  const int m_tiles = (m_rows + kBlockM - 1) / kBlockM;
  // Prefer the widest tile that still gives every SM at least one tile.
  const int cands[3] = {256, 128, 64};
  for (int i = 0; i < 3; ++i) {
    const int bn = cands[i];
    if (N % bn != 0) continue;
    const long long tiles = static_cast<long long>(m_tiles) * (N / bn);
    if (tiles < num_sms) continue;
    // With a long K a second wave of 64-column tiles that 128-column ones do not need is the dearer choice (a K block takes
    // 225 and 290 clocks).  us per launch of an fp32-sum GEMM with 64- / 128-column tiles: N = 640, K = 2560, 15 row tiles
    // 14.2 / 11.2, 24 15.2 / 11.6 (14, one wave of either: 9.2 / 11.5); N = 896, K = 3584, 11 to 20 18.4 / 13.8 to 18.9 /
    // 14.9; N = 768, K = 3072, 13 to 24 16.5 / 12.6 to 17.1 / 13.3; N = 1024, K = 4096, 10 to 18 20.0 / 14.9 to 20.7 / 15.8;
    // N = 512, K = 2048, 19 12.5 / 10.1.  (At 512, 768 and 1024 columns a forward has LayerNorm inside the GEMM by then: the
    // rule is left to the other widths and to GEMMs by themselves.)  Only where every row is valid: padded rows make no
    // tiles, and 16 sequences of up to 128 tokens, 192 tiles of 64 columns by their rows and 120 by their tokens, lost 2 %
    // of the forward with 128-column tiles.
    if (bn == 64 && all_rows && K >= 2048 && N % 128 == 0 && tiles > num_sms) return 128;
    return bn;
  }
  for (int i = 2; i >= 0; --i)
    if (N % cands[i] == 0) return cands[i];
  return 0;
}

cudaError_t launch_gemm(const GemmLaunch& g, cudaStream_t stream) {
  if (g.K % kBlockK != 0 || g.m_rows <= 0) return cudaErrorInvalidValue;
  GemmArgs a;
  a.out = g.out;
  a.bias = g.bias;
  a.residual = g.residual;
  a.m_dev = g.m_dev;
  a.m_rows = g.m_rows;
  a.N = g.N;
  a.K = g.K;
  a.status = g.status;
  a.out_ln = g.out_ln;
  a.gamma = g.gamma;
  a.beta = g.beta;
  a.gb_fp32 = g.gb_fp32 ? 1 : 0;
  a.eps = g.eps;
  a.ln_epoch = g.ln_epoch;
  a.timing = g_dbg_gemm_timing;
  // A: K-major, 128B swizzle, 8-row groups 1024 B apart; 16 K-elements = 32 B.
  a.a_desc_hi = make_smem_desc_hi(16, 1024);
  a.a_kstep_bytes = 32;
  // W: MN-major, 128B swizzle; 64-column chunks 8 KiB apart (LBO), 8-k groups
  // 1024 B apart (SBO); 16 K-rows = 2048 B.
  const uint32_t lbo = g_dbg_b_lbo ? static_cast<uint32_t>(g_dbg_b_lbo) : 64u * kBlockK * 2u;
  const uint32_t sbo = g_dbg_b_sbo ? static_cast<uint32_t>(g_dbg_b_sbo) : 1024u;
  a.b_desc_hi = make_smem_desc_hi(lbo, sbo);
  a.b_kstep_bytes = g_dbg_b_kstep ? static_cast<uint32_t>(g_dbg_b_kstep) : 2048u;
  a.split_k = 1;
  a.split_stride = 0;
  a.early_w = g_dbg_early_w != 0 ? 1 : 0;
  a.force_n = g_dbg_force_block_n >= 128 && g.N % g_dbg_force_block_n == 0 ? static_cast<int>(g_dbg_force_block_n) : 0;
  if (g.split_k > 1) {
    if (g.epilogue != BT_EPI_BIAS_RESIDUAL_F32OUT || g.N % 64 != 0 || (g.K / kBlockK) % g.split_k != 0)
      return cudaErrorInvalidValue;
    a.split_k = g.split_k;
    a.split_stride = static_cast<long long>(g.m_rows) * g.N;
    a.idesc = make_idesc_f16(kBlockM, 64, 0, 1);
    return launch_one<64, kEpiSplitKF32>(g, a, stream);
  }
  if (use_pair_kernel(g)) {
    a.idesc = make_idesc_f16(256, 256, 0, 1);  // M = 256 across the pair
    return launch_pair_epi(g, a, stream);
  }
  if (g.epilogue == BT_EPI_BIAS_RESIDUAL_LAYERNORM) return launch_ln_gemm(g, a, stream);
  int bn = g.block_n != 0 ? g.block_n : gemm_pick_block_n(g.m_rows, g.N, g.K, g.num_sms, g.all_rows);
  if (bn == 0 || g.N % bn != 0) return cudaErrorInvalidValue;
  a.idesc = make_idesc_f16(kBlockM, bn, 0, 1);
  switch (bn) {
    case 256: return launch_epi<256>(g, a, stream);
    case 128: return launch_epi<128>(g, a, stream);
    case 64: return launch_epi<64>(g, a, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace bt

// Diagnostics hook (not part of the stable ABI): overrides descriptor fields of
// the W operand / the tile width so that encodings can be compared on a device
// without rebuilding.  key: 1 = LBO bytes, 2 = SBO bytes, 3 = K-step bytes,
// 4 = forced tile width of the one-CTA kernels, 5 = pair kernel (0 auto, 1 always when
// N % 256 == 0, 2 never), 6 = programmatic dependent launch on (1, default) / off (0),
// 7 = split-K of the fp32-sum GEMMs (0 policy, < 0 never, > 0 that many K ranges),
// 8 = W blocks of a CTA's first tile requested before the dependency wait (1, default) or after (0),
// 9 = GEMM + LayerNorm on SM pairs (0, the default: by ln_pair_pays; 1 always; 2 never).
// value 0 restores the default for keys 1-5 and 7.
// Device buffer of 148 x 16 x 8 long long for clock64 stamps of the GEMM kernels (null = off):
// slots 0/1 MMA warp (accumulator free, last commit), 2/3 first epilogue warp (accumulator ready, tile
// done), 4..6 LayerNorm kernels only (4 first epilogue warp: its partials are in shared memory, 5 statistics warp 2:
// partials published, 6 first epilogue warp: mean and 1 / deviation have arrived).
extern "C" int bt_debug_set_gemm_timing(long long* device_buffer) {
  bt::g_dbg_gemm_timing = device_buffer;
  return 0;
}
// Host-side shape policies, callable without a device (tests): what 0 = tile width of the one-CTA
// kernel, 1 = K ranges of an fp32-sum GEMM, 2 = 1 if the pair kernel would take a bias-only GEMM, 3 = rows per CTA of
// LayerNorm over N columns, K partial sums, inside a forward (4: by itself), 5 = as 0 where every row is valid, 6 = 1 if GEMM +
// LayerNorm runs on SM pairs.
extern "C" int bt_debug_policy(int what, int m_rows, int N, int K, int num_sms) {
  switch (what) {
    case 0: return bt::gemm_pick_block_n(m_rows, N, K, num_sms, false);
    case 1: return bt::gemm_pick_split_k(m_rows, N, K, num_sms);
    case 5: return bt::gemm_pick_block_n(m_rows, N, K, num_sms, true);
    case 2: {
      bt::GemmLaunch g = {};
      g.m_rows = m_rows;
      g.N = N;
      g.K = K;
      g.epilogue = BT_EPI_BIAS;
      g.block_n = 0;
      g.num_sms = num_sms;
      return bt::use_pair_kernel(g) ? 1 : 0;
    }
    case 3: case 4: return bt::ln_rows_per_cta(m_rows, N, K, what == 3);
    case 6: return bt::ln_pair_pays(m_rows, N, K, num_sms) ? 1 : 0;
    default: return -1;
  }
}
extern "C" int bt_debug_set(int key, long long value) {
  switch (key) {
    case 1: bt::g_dbg_b_lbo = value; return 0;
    case 2: bt::g_dbg_b_sbo = value; return 0;
    case 3: bt::g_dbg_b_kstep = value; return 0;
    case 4: bt::g_dbg_force_block_n = value; return 0;
    case 7: bt::g_dbg_split_k = value; return 0;
    case 8: bt::g_dbg_early_w = value; return 0;
    case 9: bt::g_dbg_ln_pair = value; return 0;
    case 5: bt::g_dbg_pair_mode = value; return 0;
    case 6: bt::set_pdl_enabled(value != 0); return 0;
    default: return 1;
  }
}
