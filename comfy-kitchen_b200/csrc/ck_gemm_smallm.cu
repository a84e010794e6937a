// Block-scaled GEMMs with very few activation rows (M <= 32): weight streaming, and the one-call linears that quantize a
// dense activation of up to 16 rows inside it.
//
// out[M, N] = x[M, K] . W[N, K]^T with M small reads the whole weight once and does almost no arithmetic: it is bound
// by HBM (0.5625 bytes per NVFP4 weight element) and by fixed latencies.  The 128-row tile configurations spend their
// MMA rows, their operand loads and their epilogue on padding.  Here the operands change places: weight rows fill the
// 128 tensor-memory lanes, the activation rows are the MMA's N (32), the accumulator is 32 columns wide and the epilogue
// writes the result transposed.  Measured against the tile path: wins up to 32 rows, loses from 64 rows on.
//
// A CTA has one item; the hardware queues what does not fit the chip.  How the weight is cut (choose_plan):
//   * a 128-row tile to a CTA;
//   * few tiles and a long K: every tile's K range over a cluster of CTAs, which add their partial tiles in split order
//     through distributed shared memory.
// (Half and quarter tiles to a CTA were measured: nothing gained.  A stage, 16 KiB of weight, takes the tensor pipe some 160 cycles for its
// four MMAs, 315 with NVFP4's eight scale copies, 105 and 50 bytes a cycle: more than an SM's 24 of what HBM gives.  Four accumulators in turn
// change nothing either.)
//
// Dense activations (XT): as two kernels, the quantizer of a few rows is one wave of load latency, arithmetic and store
// latency before the GEMM's loads may begin.  Here every CTA quantizes the rows it multiplies by, stage by stage, straight
// into the shared-memory ring the tensor cores read (codes in the 128-byte swizzle, scale bytes in the tiles
// tcgen05.cp takes), while the weight's tiles come by TMA; the quantized activation never leaves the SM.  The same
// operations in the same order as quantizer + GEMM: the same bits.
//   warp 0      asks L2 for the first weight boxes ahead of the dependency wait, then TMA loads into the ring
//   warp 1      scale copies and MMAs
//   warps 2-9   dynamic tensor scale and quantizer of a dense activation (`stage_warps` of them do one stage, so that with few
//               rows several stages are in the making at once), epilogue
#include "ck_gemm_kernel.cuh"

namespace ck {
namespace {

constexpr int kMaxSmallM = 32;
constexpr int kMaxDenseM = 16;       // rows that are quantized here (which of them by format: linear_small_m_applies)
constexpr int kMmaN = 32;            // of the MMA: activation rows; those past M are whatever the ring holds, their columns are not read
constexpr int kQuantWarps = 8;
constexpr int kSmallThreads = 64 + 32 * kQuantWarps;
constexpr int kMaxSmemBytes = 224 * 1024;  // of a CTA alone on its SM

struct SmallParams {
  const void* x;             // dense activation [M, K], or null: quantized, and
  const uint8_t* x_scales;   //   its tiled block scales
  const float* x_scale;      // tensor scale of the activation (NVFP4); of a dense one the static scale, or null: from
  const float* partials;     //   the maxima of a reduction pass, or without them
  int n_partials;
  int n_vecs;                //   from x itself, n_vecs 32-byte units that every CTA reads
  const uint8_t* w_scales;   // tiled block scales of the weight
  const float* w_scale;      // its tensor scale (NVFP4)
  const float* alpha;        // replaces the product of the tensor scales when non-null
  const void* bias;
  void* out;                 // [M, N]
  int bias_dtype, out_dtype;
  int M, N, K;
  int k_bytes, sf_col_tiles;
  int splits, k_stages_per_split;
  int ring;                  // stages of the ring
  int x_rows;                // activation rows of a stage's slot: 16 or 32
  int prefetch;              // weight boxes asked from L2 ahead of the dependency wait
  int stage_warps;           // dense: quantizer warps to a stage, 2, 4 or 8
  int* status;
};

template <Kind KIND>
struct Small {
  static constexpr int kSfTiles = KIND == Kind::kNvfp4 ? 4 : 1;
  static constexpr int kSfBytes = kSfTiles * 512;
  static constexpr int kMaxRing = 7;
  static constexpr int kSfCols = 2 * kSfTiles * 4;  // tensor-memory columns of a stage's scales
  static constexpr int kTmemCols = pow2_at_least(kMmaN + kMaxRing * kSfCols);
  static constexpr int kStageElems = KIND == Kind::kNvfp4 ? 2 * kStageKBytes : kStageKBytes;
  static constexpr int kRowThreads = kStageElems / 16;  // a thread takes 16 elements of a row
  static constexpr uint32_t kIdesc = make_block_scaled_idesc(KIND == Kind::kNvfp4 ? 1u : 0u, KIND == Kind::kNvfp4 ? 0u : 1u, kTileM, kMmaN);
  static_assert(kTmemCols <= 256, "two CTAs to an SM");
  static_assert(kMaxDenseM * kRowThreads <= 32 * kQuantWarps, "a stage's rows in one go");
  // The ring: weight [ring][128 rows x 128 bytes], activation codes [ring][x_rows x 128 bytes], scale tiles of both.  (An MMA
  // reads 32 activation rows: with slots of 16 into what follows.)
  static constexpr int smem_bytes(int ring, int x_rows) {
    return ring * ((kTileM + x_rows) * kStageKBytes + 2 * kSfBytes) + 1024 /*alignment slack*/;
  }
  static_assert(2 * 4 * kSfBytes >= 16 * kStageKBytes, "what a slot of 16 rows lacks");
  static_assert(kMaxSmallM * kTileM * 4 <= 4 * kTileM * kStageKBytes, "a partial tile fits in the weight's slots");
};

template <typename T>
__device__ __forceinline__ quant::Sixteen<T> load_sixteen(const T* p, bool valid) {
  quant::Sixteen<T> r = {};
  if (valid) {
#pragma unroll
    for (int h = 0; h < static_cast<int>(sizeof(T)) / 2; ++h) {
      const Vec256 v = ld_global_stream_256(p + 8 * h);
#pragma unroll
      for (int i = 0; i < 8; ++i) r.w[8 * h + i] = v.w[i];
    }
  }
  return r;
}

// amax(|x|) / 2688 by the quantizer warps (all of them return it)
template <typename T>
__device__ __forceinline__ float dynamic_scale(const SmallParams& p, int tid, float* warp_max) {
  constexpr int kThreads = 32 * kQuantWarps;
  constexpr int kInFlight = 8;
  float m = 0.0f;
  if (p.n_partials > 0) {
    for (int i = tid; i < p.n_partials; i += kThreads) m = fmaxf(m, ld_f32_dependent(p.partials + i));
  } else {
    const T* x = static_cast<const T*>(p.x);
    for (int i = tid; i < p.n_vecs; i += kInFlight * kThreads) {
      Vec256 raw[kInFlight];
#pragma unroll
      for (int j = 0; j < kInFlight; ++j) {
        raw[j] = i + j * kThreads < p.n_vecs ? ld_global_stream_256(x + (i + j * kThreads) * (32 / sizeof(T))) : Vec256{};
      }
#pragma unroll
      for (int j = 0; j < kInFlight; ++j) m = fmaxf(m, quant::abs_max_of_vec<T>(raw[j]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if ((tid & 31) == 0) warp_max[tid >> 5] = m;
  named_barrier_sync(1, kThreads);
#pragma unroll
  for (int w = 0; w < kQuantWarps; ++w) m = fmaxf(m, warp_max[w]);
  return quant::nvfp4_scale_of_amax<T>(m);
}

// Position in the ring: `step` moves on by up to a round.
struct RingAt {
  int slot;
  uint32_t phase;
  __device__ explicit RingAt(int first) : slot(first), phase(0) {}
  __device__ __forceinline__ void step(int by, int ring) {
    slot += by;
    if (slot >= ring) {
      slot -= ring;
      phase ^= 1u;
    }
  }
};

template <typename OutT>
__device__ __forceinline__ void store_columns(OutT* dst, int64_t pitch, const uint32_t (&acc)[16], float alpha, float bias, int count) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (i < count) *dst = to_out<OutT>(fmaf(__uint_as_float(acc[i]), alpha, bias));
    dst += pitch;
  }
}

// The cluster's share of one weight tile: partial tiles lie in the CTAs' shared memory as [activation row][128].
template <typename OutT>
__device__ __forceinline__ void add_cluster_tile(const SmallParams& p, OutT* out, const uint32_t (&base)[kMaxSplits], int rank, int qw,
                                                 int lane, int n0, float alpha) {
  if (4 * p.M <= p.splits * kQuantWarps) {  // a warp to 32 weight rows of one activation row, if there are warps enough
    const int u = rank + p.splits * qw, m = u >> 2, r = (u & 3) * 32 + lane, n = n0 + r;
    if (m < p.M) {
      float v[kMaxSplits];
#pragma unroll
      for (int i = 0; i < kMaxSplits; ++i) {
        if (i < p.splits) v[i] = ld_shared_cluster_f32(base[i] + (m * kTileM + r) * 4);
      }
      float acc = v[0];
#pragma unroll
      for (int i = 1; i < kMaxSplits; ++i) {
        if (i < p.splits) acc += v[i];
      }
      if (n < p.N) {
        const float bias = p.bias != nullptr ? load_bias(p.bias, p.bias_dtype, n) : 0.0f;
        out[static_cast<int64_t>(m) * p.N + n] = to_out<OutT>(fmaf(acc, alpha, bias));
      }
    }
    return;
  }
  // else all 128 weight rows, a lane four of them (NVFP4 32 x 1024 x 4096: 5.8 us, against 7.1 with 32 weight rows at a time)
  const int n = n0 + lane * 4;
  const bool inside = n < p.N;  // N % 8 == 0: all four or none
  const bool vec = (reinterpret_cast<uintptr_t>(out) & (4 * sizeof(OutT) - 1)) == 0;
  float bias[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (p.bias != nullptr && inside) {
#pragma unroll
    for (int j = 0; j < 4; ++j) bias[j] = load_bias(p.bias, p.bias_dtype, n + j);
  }
  for (int m = rank + p.splits * qw; m < p.M; m += p.splits * kQuantWarps) {
    const float4 acc = add_partials(base, p.splits, (m * kTileM + lane * 4) * 4);
    if (inside) {
      float y[4];
      sums_scaled(acc, alpha, bias, y);
      OutT* dst = out + static_cast<int64_t>(m) * p.N + n;
      if (vec) {
        store_four(dst, y);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[j] = to_out<OutT>(y[j]);
      }
    }
  }
}

template <Kind KIND, typename XT, bool SPLIT>
__global__ void __launch_bounds__(kSmallThreads, 2)
small_m_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const SmallParams p) {
  using C = Small<KIND>;
  constexpr bool kDense = !std::is_void<XT>::value;
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kABytes = kTileM * kStageKBytes;
  const int b_bytes = p.x_rows * kStageKBytes;
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem_a + p.ring * kABytes;
  uint8_t* smem_sfa = smem_b + p.ring * b_bytes;
  uint8_t* smem_sfb = smem_sfa + p.ring * C::kSfBytes;
  __shared__ uint64_t full_bar[C::kMaxRing];   // loads landed and rows quantized -> MMA
  __shared__ uint64_t empty_bar[C::kMaxRing];  // MMA -> producer and quantizers
  __shared__ uint64_t acc_bar[1];
  __shared__ uint32_t tmem_base_slot[1];
  __shared__ int abort_word;
  __shared__ float warp_max[kQuantWarps];
  volatile int* abort_flag = &abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = SPLIT ? blockIdx.x : 0;
  const int n0 = blockIdx.y * kTileM;  // this tile's weight rows
  const int k_stages = (p.k_bytes + kStageKBytes - 1) / kStageKBytes;
  const int ks0 = rank * p.k_stages_per_split;
  const int n_stages = min(k_stages - ks0, p.k_stages_per_split);
  const uint8_t* w_scales = p.w_scales + (static_cast<int64_t>(blockIdx.y) * p.sf_col_tiles + ks0 * C::kSfTiles) * 512;
  const int sf_tiles = min(p.sf_col_tiles - ks0 * C::kSfTiles, n_stages * C::kSfTiles);  // of this CTA's K range

  uint32_t tmem_base = 0;
  if (warp == 0) {
    if (elect_one()) {
      // A prefetch only warms L2 (the point of coherence): it may run ahead of the kernel before this one.
      for (int i = 0; i < min(n_stages, p.prefetch); ++i) {
        tma_prefetch_2d(&map_w, (ks0 + i) * kStageKBytes, n0);
        if constexpr (!kDense) tma_prefetch_2d(&map_x, (ks0 + i) * kStageKBytes, 0);
      }
      if (p.prefetch > 0) bulk_prefetch_l2(w_scales, static_cast<uint32_t>(min(sf_tiles, p.prefetch * C::kSfTiles)) * 512u);
      *abort_flag = 0;
      for (int s = 0; s < p.ring; ++s) {
        mbar_init(&full_bar[s], kDense ? 1 + p.stage_warps : 1);
        mbar_init(&empty_bar[s], 1);
      }
      mbar_init(acc_bar, 1);
      fence_barrier_init();
      __threadfence_block();
    }
    __syncwarp();
    named_barrier_arrive(2, kSmallThreads);
  } else {
    if (warp == 1) {
      tmem_alloc<1>(tmem_base_slot, C::kTmemCols);
    } else if constexpr (kDense) {
      // the rows of this CTA's K range: one 128-byte line per thread and step
      const int lines = (n_stages * C::kStageElems * static_cast<int>(sizeof(XT)) + 127) / 128;
      const int pitch = p.K * static_cast<int>(sizeof(XT));
      const int first = ks0 * C::kStageElems * static_cast<int>(sizeof(XT));
      for (int m = warp - 2; m < p.M; m += kQuantWarps) {
        for (int l = lane; l < lines; l += 32) {
          if (first + l * 128 < pitch) prefetch_l2(static_cast<const uint8_t*>(p.x) + static_cast<int64_t>(m) * pitch + first + l * 128);
        }
      }
    }
    tc_fence_before_sync();
    named_barrier_sync(2, kSmallThreads);
    tc_fence_after_sync();
    tmem_base = *tmem_base_slot;
  }

  float alpha = 1.0f;  // quantizer warps
  if (warp == 0) {
    // ------------------------------------------------------------------ weight loads
    if (elect_one()) {  // for the whole loop: see ck_gemm_kernel.cuh
      const uint32_t full_addr = smem_u32(full_bar), empty_addr = smem_u32(empty_bar);
      const uint32_t a_addr = smem_u32(smem_a), b_addr = smem_u32(smem_b), sfa_addr = smem_u32(smem_sfa), sfb_addr = smem_u32(smem_sfb);
      const uint8_t* x_scales = p.x_scales + static_cast<int64_t>(ks0) * C::kSfTiles * 512;
      RingAt at(0);
      for (int i = 0; i < n_stages; ++i, at.step(1, p.ring)) {
        const int s = at.slot;
        const uint32_t bar = full_addr + s * 8;
        mbar_wait(empty_addr + s * 8, at.phase ^ 1, abort_flag);
        const uint32_t sf_bytes = static_cast<uint32_t>(min(C::kSfTiles, sf_tiles - i * C::kSfTiles)) * 512u;
        mbar_arrive_expect_tx(bar, kDense ? kABytes + sf_bytes : kABytes + p.M * kStageKBytes + 2 * sf_bytes);
        if (i == 0) pdl_wait();
        tma_load_2d(a_addr + s * kABytes, &map_w, bar, (ks0 + i) * kStageKBytes, n0);
        bulk_load_1d(sfa_addr + s * C::kSfBytes, w_scales + static_cast<int64_t>(i) * C::kSfTiles * 512, sf_bytes, bar);
        if constexpr (!kDense) {
          tma_load_2d(b_addr + s * b_bytes, &map_x, bar, (ks0 + i) * kStageKBytes, 0);
          bulk_load_1d(sfb_addr + s * C::kSfBytes, x_scales + static_cast<int64_t>(i) * C::kSfTiles * 512, sf_bytes, bar);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    pdl_wait();  // see ck_gemm_kernel.cuh: keeps the bounded waits from running out behind a long predecessor
    if (elect_one()) {
      const uint32_t full_addr = smem_u32(full_bar), empty_addr = smem_u32(empty_bar);
      const uint32_t a_lo0 = static_cast<uint32_t>(make_operand_desc_sw128(smem_u32(smem_a)));
      const uint32_t b_lo0 = static_cast<uint32_t>(make_operand_desc_sw128(smem_u32(smem_b)));
      const uint32_t op_hi = static_cast<uint32_t>(make_operand_desc_sw128(0) >> 32);
      const uint32_t sfa_lo0 = static_cast<uint32_t>(make_scale_desc(smem_u32(smem_sfa)));
      const uint32_t sfb_lo0 = static_cast<uint32_t>(make_scale_desc(smem_u32(smem_sfb)));
      const uint32_t sf_hi = static_cast<uint32_t>(make_scale_desc(0) >> 32);
      const int total_mma = (p.k_bytes + kMmaKBytes - 1) / kMmaKBytes - ks0 * kMmaPerStage;
      RingAt at(0);
      for (int i = 0; i < n_stages; ++i, at.step(1, p.ring)) {
        const int s = at.slot;
        mbar_wait(full_addr + s * 8, at.phase, abort_flag);
        tc_fence_after_sync();
        const uint32_t t_sfa = tmem_base + kMmaN + s * C::kSfCols, t_sfb = t_sfa + C::kSfTiles * 4;
#pragma unroll
        for (int t = 0; t < C::kSfTiles; ++t) {
          tc_copy_scales_32x128b<1>(t_sfa + t * 4, desc64(sfa_lo0 + s * (C::kSfBytes >> 4) + t * 32, sf_hi));
          tc_copy_scales_32x128b<1>(t_sfb + t * 4, desc64(sfb_lo0 + s * (C::kSfBytes >> 4) + t * 32, sf_hi));
        }
        auto mma = [&](int kb) {
          const uint32_t accumulate = (i != 0 || kb != 0) ? 1u : 0u;
          const uint64_t a_desc = desc64(a_lo0 + s * (kABytes >> 4) + kb * 2, op_hi);
          const uint64_t b_desc = desc64(b_lo0 + s * (b_bytes >> 4) + kb * 2, op_hi);
          if constexpr (KIND == Kind::kNvfp4) {
            mma_nvfp4<1>(tmem_base, a_desc, b_desc, C::kIdesc, t_sfa + kb * 4, t_sfb + kb * 4, accumulate);
          } else {
            mma_mxfp8<1>(tmem_base, a_desc, b_desc, idesc_with_scale_ids(C::kIdesc, kb), t_sfa, t_sfb, accumulate);
          }
        };
        const int n_mma = total_mma - i * kMmaPerStage;  // left from here on
        // one straight path for whole stages and the last one: a loop of its own for the last (code met once, and cold) cost more than the
        // predicates (us: bf16 24 x 9216 x 3072 5.7 / 5.4, 8 x 18432 x 3072 with x dense 8.9 / 8.7, fp32 1 x 3072 x 3072 5.8 / 5.1, 4 x 6208 x 896 4.4 / 4.2)
#pragma unroll
        for (int kb = 0; kb < kMmaPerStage; ++kb) {
          if (kb < n_mma) mma(kb);
        }
        tc_commit<1>(empty_addr + s * 8);
        if (i == n_stages - 1) tc_commit<1>(smem_u32(acc_bar));
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ quantizer, epilogue
    pdl_wait();
    const int qw = warp - 2, qt = threadIdx.x - 64;
    if constexpr (kDense) {
      float g = 1.0f;
      if constexpr (KIND == Kind::kNvfp4) {
        g = p.x_scale != nullptr ? ld_f32_dependent(p.x_scale) : dynamic_scale<XT>(p, qt, warp_max);
        alpha = g * ld_f32_dependent(p.w_scale);
      }
      [[maybe_unused]] const quant::TensorScale ts = quant::make_tensor_scale(g);
      // A group of stage_warps warps does every groups-th stage.  No more groups than slots: when a group comes to a stage, the
      // one two rounds before it in its slot has then been used up (a wait by parity cannot tell a phase from the one two later).
      const int groups = kQuantWarps / p.stage_warps;
      const int group = qw / p.stage_warps, t_in_group = (qw % p.stage_warps) * 32 + lane;
      const int unit = t_in_group % C::kRowThreads, row = t_in_group / C::kRowThreads;  // 16 elements of a row of the stage
      const bool in_rows = row < p.M;
      // threads past the last row take the first one's elements (nothing slow like a division of zeros) and write nothing
      const XT* x = static_cast<const XT*>(p.x) + static_cast<int64_t>(in_rows ? row : 0) * p.K + static_cast<int64_t>(ks0) * C::kStageElems + unit * 16;
      const int cols = p.K - ks0 * C::kStageElems - unit * 16;  // columns left from this thread's first element on
      auto load_stage = [&](int i) { return load_sixteen<XT>(x + i * C::kStageElems, i < n_stages && i * C::kStageElems < cols); };
      const uint32_t data_at = row * kStageKBytes + (KIND == Kind::kNvfp4 ? (((unit >> 1) ^ (row & 7)) << 4) + (unit & 1) * 8 : (unit ^ (row & 7)) << 4);
      const uint32_t scale_at = row * 16 + (KIND == Kind::kNvfp4 ? (unit >> 2) * 512 + (unit & 3) : unit >> 1);
      quant::Sixteen<XT> next = load_stage(group), after = load_stage(group + groups);  // the loads run two stages ahead
      RingAt at(group);
      for (int i = group; i < n_stages; i += groups, at.step(groups, p.ring)) {
        const int s = at.slot;
        const quant::Sixteen<XT> now = next;
        next = after;
        after = load_stage(i + 2 * groups);
        if constexpr (KIND == Kind::kNvfp4) {
          const quant::Sixteen<XT> one[1] = {now};
          uint32_t codes[1][2], byte[1];
          quant::nvfp4_blocks<XT, true, 1>(one, ts, codes, byte);
          uint32_t lo = codes[0][0], hi = codes[0][1], scale = byte[0];
          if (i * C::kStageElems >= cols) lo = hi = scale = 0;  // past K: the last MMA may reach there
          mbar_wait(&empty_bar[s], at.phase ^ 1, abort_flag);
          if (in_rows) {
            *reinterpret_cast<uint2*>(smem_b + s * b_bytes + data_at) = make_uint2(lo, hi);
            smem_sfb[s * C::kSfBytes + scale_at] = static_cast<uint8_t>(scale);
          }
        } else {
          float v[16];
          now.widen(v);
          float amax = quant::amax16(v);
          amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));  // the block's other half
          const quant::Mxfp8Scale sc = quant::mxfp8_scale(amax);
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) w[j] = quant::mxfp8_four(v + 4 * j, sc);
          mbar_wait(&empty_bar[s], at.phase ^ 1, abort_flag);
          if (in_rows) {
            *reinterpret_cast<uint4*>(smem_b + s * b_bytes + data_at) = make_uint4(w[0], w[1], w[2], w[3]);
            if ((unit & 1) == 0) smem_sfb[s * C::kSfBytes + scale_at] = static_cast<uint8_t>(sc.byte);
          }
        }
        fence_proxy_async();  // what was written becomes visible to the tensor cores' reads
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[s]);
      }
    } else {
      if (p.alpha != nullptr) {
        alpha = ld_f32_dependent(p.alpha);
      } else if (p.x_scale != nullptr && p.w_scale != nullptr) {
        alpha = ld_f32_dependent(p.x_scale) * ld_f32_dependent(p.w_scale);
      }
    }
    // ---- epilogue: lane = weight row (output column), accumulator columns = activation rows, 16 to a warp
    const int quarter = warp & 3, m0 = (qw >> 2) * 16;
    const int r = quarter * 32 + lane, n = n0 + r;
    if (m0 < p.M) {
      float bias = 0.0f;
      if (!SPLIT && p.bias != nullptr && n < p.N) bias = load_bias(p.bias, p.bias_dtype, n);
      mbar_wait(acc_bar, 0, abort_flag);
      tc_fence_after_sync();
      uint32_t acc[16];
      tmem_load_32x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + m0, acc);
      tmem_load_wait();
      if constexpr (SPLIT) {
        float* partial = reinterpret_cast<float*>(smem) + m0 * kTileM + r;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          if (m0 + c < p.M) partial[c * kTileM] = __uint_as_float(acc[c]);
        }
      } else if (n < p.N) {
        const int64_t at = static_cast<int64_t>(m0) * p.N + n;
        switch (p.out_dtype) {
          case CK_DTYPE_BF16: store_columns(static_cast<__nv_bfloat16*>(p.out) + at, p.N, acc, alpha, bias, p.M - m0); break;
          case CK_DTYPE_F16: store_columns(static_cast<__half*>(p.out) + at, p.N, acc, alpha, bias, p.M - m0); break;
          default: store_columns(static_cast<float*>(p.out) + at, p.N, acc, alpha, bias, p.M - m0);
        }
      }
    }
  }

  if constexpr (SPLIT) {
    // the CTAs of the cluster add their partial tiles in split order (ck_gemm_kernel.cuh)
    __syncwarp();
    cluster_sync_all();
    if (warp >= 2) {
      uint32_t base[kMaxSplits];
#pragma unroll
      for (int i = 0; i < kMaxSplits; ++i) base[i] = map_to_cta(smem_u32(smem), i < p.splits ? i : 0);
      switch (p.out_dtype) {
        case CK_DTYPE_BF16: add_cluster_tile(p, static_cast<__nv_bfloat16*>(p.out), base, rank, warp - 2, lane, n0, alpha); break;
        case CK_DTYPE_F16: add_cluster_tile(p, static_cast<__half*>(p.out), base, rank, warp - 2, lane, n0, alpha); break;
        default: add_cluster_tile(p, static_cast<float*>(p.out), base, rank, warp - 2, lane, n0, alpha);
      }
    }
    __syncwarp();
    cluster_sync_all();  // no CTA leaves while another may still read its partial
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicExch(p.status, 1);
    // give copies that may still be in flight time to land before the CTA's memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, C::kTmemCols);
  }
}

struct SmallPlan {
  int splits;        // CTAs that share a tile's K range
  bool two_per_sm;   // some SMs get two CTAs at once
};

// Clusters of `splits` CTAs that run at once with one CTA on an SM (the request for shared memory sees to that).
template <Kind KIND>
int clusters_of(int splits, int* out) {
  static std::atomic<int> cached[64][kMaxSplits + 1];
  int dev = 0;
  CK_CUDA(cudaGetDevice(&dev));
  int n = (dev >= 0 && dev < 64) ? cached[dev][splits].load(std::memory_order_relaxed) : 0;
  if (n == 0) {
    constexpr int kMoreThanHalf = 128 * 1024;
    auto kernel = small_m_kernel<KIND, void, true>;
    CK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemBytes));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kSmallThreads);
    cfg.gridDim = dim3(static_cast<unsigned>(splits), static_cast<unsigned>(sm_count() / splits));
    cfg.dynamicSmemBytes = kMoreThanHalf;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CK_CUDA(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
    if (n < 1) n = 1;
    if (dev >= 0 && dev < 64) cached[dev][splits].store(n, std::memory_order_relaxed);
  }
  *out = n;
  return CK_OK;
}

// CTAs per tile (1 = no split).  The most whose clusters all run at once with one CTA on an SM; with two on an SM
// when that leaves a CTA more than ten stages.  (A cluster that finds no room runs later: nobody waits for
// it.)  Graph replays, us, few CTAs of many stages / more: NVFP4 32 x 4096 x 12288 (12 stages / 8) 8.9 / 8.0,
// 1 x 6144 x 8192 (16 / 7) 8.9 / 8.1, 1 x 6144 x 6144 (12 / 5) 7.6 / 7.6, MXFP8 32 x 6144 x 12288 (48 / 20) 18.3 / 11.7,
// 1 x 4096 x 12288 (24 / 16) 10.9 / 9.6; but NVFP4 1 x 4096 x 8192 (8 / 6) 6.6 / 7.1, 1 x 6144 x 4096 (8 / 4) 6.2 / 6.4.
template <Kind KIND>
int choose_plan(int64_t N, int k_bytes, SmallPlan* plan) {
  const int k_stages = static_cast<int>(ceil_div(k_bytes, kStageKBytes));
  const int64_t tiles = ceil_div(N, kTileM);
  const int most = small_m_max_splits(N, k_bytes);
  constexpr int kMaxStagesAlone = 10;
  int splits = 1;
  for (int per_sm = 1; per_sm <= 2; ++per_sm) {
    for (splits = most; splits > 1; --splits) {
      int clusters = 0;
      if (int rc = clusters_of<KIND>(splits, &clusters)) return rc;
      if (clusters * per_sm >= tiles) break;
    }
    if (ceil_div(k_stages, splits) <= kMaxStagesAlone) break;
  }
  plan->splits = static_cast<int>(ceil_div(k_stages, ceil_div(k_stages, splits)));  // none without a stage
  int alone = 0;
  if (int rc = clusters_of<KIND>(plan->splits, &alone)) return rc;
  plan->two_per_sm = tiles > alone;
  return CK_OK;
}

template <Kind KIND, typename XT, bool SPLIT>
int launch_as(const void* w, const void* codes, const SmallParams& p, cudaStream_t stream) {
  using C = Small<KIND>;
  auto kernel = small_m_kernel<KIND, XT, SPLIT>;
  CUtensorMap map_w, map_x = {};
  if (int rc = make_operand_map(&map_w, w, p.N, p.k_bytes, kTileM)) return rc;
  if (std::is_void<XT>::value) {
    // no rows past M in a box: filling them costs (us: NVFP4 1 x 5120 x 9216 8.0 / 7.6, MXFP8 4 x 3072 x 3072 5.4 / 5.2)
    if (int rc = make_operand_map(&map_x, codes, p.M, p.k_bytes, p.M)) return rc;
  }
  const int smem = C::smem_bytes(p.ring, p.x_rows);
  static std::atomic<bool> configured[64];
  int dev = 0;
  CK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    CK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemBytes));
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.splits), static_cast<unsigned>(ceil_div(p.N, kTileM)));
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attrs = 0;
  if (SPLIT) {
    attr[n_attrs].id = cudaLaunchAttributeClusterDimension;
    attr[n_attrs].val.clusterDim.x = p.splits;
    attr[n_attrs].val.clusterDim.y = 1;
    attr[n_attrs++].val.clusterDim.z = 1;
  }
  if (pdl_enabled()) {
    attr[n_attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attrs;
  CK_CUDA(cudaLaunchKernelEx(&cfg, kernel, map_w, map_x, p));
  return CK_OK;
}

template <Kind KIND, typename XT>
int launch(const void* w, const void* codes, SmallParams p, cudaStream_t stream) {
  SmallPlan plan = {};
  if (int rc = choose_plan<KIND>(p.N, p.k_bytes, &plan)) return rc;
  p.splits = plan.splits;
  p.k_stages_per_split = static_cast<int>(ceil_div(ceil_div(p.k_bytes, kStageKBytes), p.splits));
  p.x_rows = p.M <= 16 ? 16 : 32;
  constexpr int kTwoToAnSm = 228 * 1024 / 2 - 1024 /*reserved*/ - 512 /*barriers, maxima*/;
  static_assert(Small<KIND>::smem_bytes(5, 16) <= kTwoToAnSm && Small<KIND>::smem_bytes(4, 32) <= kTwoToAnSm, "two CTAs to an SM");
  static_assert(Small<KIND>::smem_bytes(7, 32) <= kMaxSmemBytes, "one CTA to an SM");
  // Alone on its SM a CTA gets all the stages that tensor memory has columns for; where two share an SM, what leaves room for
  // both (MXFP8 8 x 18432 x 6144, us: four stages 22.7, five 21.9, seven 20.5; NVFP4 16 x 18432 x 12288 24.1 / 23.5 / 22.0, 8 x 9216
  // x 3072 6.40 / 6.13 / 5.92; but MXFP8 8 x 3072 x 12288, eight CTAs to a tile, 10.4 / 10.3 / 15.3).
  p.ring = !plan.two_per_sm ? 7 : p.x_rows == 16 ? 5 : 4;
  // Weight boxes asked from L2 ahead of the dependency wait.  Few: the requests queue in front of the loads in the TMA unit
  // (NVFP4 8 x 18432 x 3072 from a dense activation: none 8.56 us, two 8.41, four 8.69, sixteen 9.44; lines asked by the idle
  // quantizer threads instead, twelve boxes' worth, 9.81; quantized, sixteen instead of four 10.4 against 8.9).
  p.prefetch = std::is_void<XT>::value ? 4 : 2;
  // a thread takes 16 elements: 16 (NVFP4) or 8 (MXFP8) threads to a row of a stage
  const int stage_warps = static_cast<int>(ceil_div(p.M * Small<KIND>::kRowThreads, 32));
  p.stage_warps = stage_warps <= 2 ? 2 : stage_warps <= 4 ? 4 : 8;
  if (int rc = gemm_status_word(&p.status)) return rc;
  return p.splits > 1 ? launch_as<KIND, XT, true>(w, codes, p, stream) : launch_as<KIND, XT, false>(w, codes, p, stream);
}

template <typename XT>
int launch(bool is_mxfp8, const void* w, const void* codes, const SmallParams& p, cudaStream_t s) {
  return is_mxfp8 ? launch<Kind::kMxfp8, XT>(w, codes, p, s) : launch<Kind::kNvfp4, XT>(w, codes, p, s);
}

SmallParams params_of(bool is_mxfp8, const void* w_scales, const float* w_scale, const void* bias, int bias_dtype, void* out, int out_dtype, int64_t M,
                      int64_t N, int64_t K) {
  SmallParams p{};
  p.w_scales = static_cast<const uint8_t*>(w_scales);
  p.w_scale = w_scale;
  p.bias = bias;
  p.out = out;
  p.bias_dtype = bias_dtype;
  p.out_dtype = out_dtype;
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.K = static_cast<int>(K);
  p.k_bytes = static_cast<int>(is_mxfp8 ? K : K / 2);
  p.sf_col_tiles = static_cast<int>(ceil_div(K / (is_mxfp8 ? 32 : 16), 4));
  return p;
}

}  // namespace

bool small_m_applies(int64_t M, int64_t N, int64_t K) { return M >= 1 && M <= kMaxSmallM && N >= 1 && N <= 65535ll * kTileM && K >= 32; }

// CTAs per 128-row weight tile (1 = no split): as many as let two CTAs run on every SM and leave each
// of them four pipeline stages.
int small_m_max_splits(int64_t N, int k_bytes) {
  const int k_stages = static_cast<int>(ceil_div(k_bytes, kStageKBytes));
  const int64_t tiles = ceil_div(N, kTileM);
  if (tiles * 3 > sm_count() || k_stages < 16) return 1;
  int splits = min(kMaxSplits, k_stages / 4);
  const int64_t by_sms = 2 * static_cast<int64_t>(sm_count()) / tiles;
  if (by_sms < splits) splits = static_cast<int>(by_sms);
  return max(splits, 1);
}

int small_m_splits(bool is_mxfp8, int64_t N, int k_bytes, int* splits) {
  SmallPlan plan = {};
  const int rc = is_mxfp8 ? choose_plan<Kind::kMxfp8>(N, k_bytes, &plan) : choose_plan<Kind::kNvfp4>(N, k_bytes, &plan);
  *splits = plan.splits;
  return rc;
}

// a: activation [M, K], b: weight [N, K] (the public argument order); shapes and pointers were validated by the caller.
int scaled_mm_small_m(bool is_mxfp8, const void* a, const void* b, const void* sfa, const void* sfb, const float* tsa,
                      const float* tsb, const float* alpha, const void* bias, int bias_dtype, void* out, int out_dtype,
                      int64_t M, int64_t N, int64_t K, cudaStream_t stream) {
  SmallParams p = params_of(is_mxfp8, sfb, tsb, bias, bias_dtype, out, out_dtype, M, N, K);
  p.x_scales = static_cast<const uint8_t*>(sfa);
  p.x_scale = tsa;
  p.alpha = alpha;
  return launch<void>(is_mxfp8, b, a, p, stream);
}

// What is quantized inside the GEMM; everything else, wrong arguments among it, is left to the separate calls.
bool linear_small_m_applies(bool is_mxfp8, const void* x, int x_dtype, const void* w, const void* w_scales, int bias_dtype, const void* out,
                            int out_dtype, int64_t M, int64_t N, int64_t K) {
  auto aligned = [](const void* p, uintptr_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; };
  auto is_float = [](int dtype) { return dtype == CK_DTYPE_F32 || dtype == CK_DTYPE_F16 || dtype == CK_DTYPE_BF16; };
  // Up to 8 rows of NVFP4 and 16 of MXFP8, whose rows take half the threads, the quantizer's warps keep up with the stream.
  // Quantizer + GEMM / one kernel, us: NVFP4 static scale 8 x 18432 x 3072 9.9 / 8.5, 8 x 3072 x 3072 8.0 / 6.6, but 10 x 3072 x 3072 8.7 / 9.2,
  // 16 x 6144 x 3072 9.2 / 10.2; MXFP8 16 x 3072 x 3072 7.3 / 5.8, 16 x 18432 x 12288 42.8 / 41.9.
  const int64_t limit = is_mxfp8 ? 16 : 8;
  const int forced = forced_gemm_config();
  // A result written over its own activation is for the separate kernels: here every CTA reads all of x until it ends.
  const uintptr_t x0 = reinterpret_cast<uintptr_t>(x), out0 = reinterpret_cast<uintptr_t>(out);
  auto bytes = [](int dtype, int64_t n) { return static_cast<uintptr_t>(n) * (dtype == CK_DTYPE_F32 ? 4 : 2); };
  const bool apart = x0 + bytes(x_dtype, M * K) <= out0 || out0 + bytes(out_dtype, M * N) <= x0;
  return apart && M <= limit && small_m_applies(M, N, K) && N % 8 == 0 && K % 32 == 0 && K <= (1 << 28) && is_float(x_dtype) && is_float(out_dtype) &&
         is_float(bias_dtype) && aligned(x, 32) && aligned(w, 16) && aligned(w_scales, 16) && !exact_division() && (forced == 0 || forced == 9);
}

// NVFP4 with a dynamic scale: whether every CTA takes the maximum of the whole activation itself, or a reduction kernel leaves partial
// maxima: by the activation's bytes.  us, reduction kernel / whole activation: CTAs alone on their SMs bf16 6 x 3072 x 6144 (72 KiB) 7.8 / 7.4, 8 x 3072 x 6144
// (96 KiB) 7.8 / 7.6, 4 x 3072 x 12288 (96 KiB) 9.4 / 9.2, fp32 8 x 6144 x 4096 (128 KiB) 9.4 / 8.9, bf16 6 x 3072 x 12288 (144 KiB) 9.6 / 10.1, 8 x
// 12288 x 15360 (240 KiB) 23.8 / 25.0.  Where two share an SM, both want the whole activation at once: bf16 4 x 5120 x 9216 (72 KiB) 9.9 / 10.6, 6 x
// 6144 x 8512 (100 KiB) 10.8 / 11.8, 8 x 24576 x 8128 (127 KiB) 23.5 / 25.2, fp16 2 x 4096 x 25600 (100 KiB) 15.5 / 15.8; fp32 has half the elements
// to look at: 2 x 5120 x 9216 (72 KiB) 10.2 / 9.9, 2 x 6144 x 12800 (100 KiB) 13.2 / 12.8, 4 x 5120 x 8128 (127 KiB) 10.3 / 10.6, 8 x 24576 x 4032
// 16.6 / 17.5.
int linear_small_m_reads_whole_input(int x_dtype, int64_t M, int64_t N, int64_t K, bool* whole) {
  constexpr int64_t kShared = 64 * 1024, kSharedFp32 = 112 * 1024, kAlone = 128 * 1024;
  const bool fp32 = x_dtype == CK_DTYPE_F32;
  const int64_t bytes = M * K * (fp32 ? 4 : 2), shared = fp32 ? kSharedFp32 : kShared;
  *whole = bytes <= kAlone;
  if (bytes <= shared || !*whole) return CK_OK;  // whatever the plan
  SmallPlan plan = {};
  if (int rc = choose_plan<Kind::kNvfp4>(N, static_cast<int>(K / 2), &plan)) return rc;
  *whole = !plan.two_per_sm;
  return CK_OK;
}

// `partials`: maxima of a reduction pass for a dynamic scale, or null (every CTA reads all of x).
int linear_small_m(bool is_mxfp8, const void* x, int x_dtype, const float* x_scale, const float* partials, int n_partials, const void* w,
                   const void* w_scales, const float* w_scale, const void* bias, int bias_dtype, void* out, int out_dtype, int64_t M,
                   int64_t N, int64_t K, cudaStream_t stream) {
  SmallParams p = params_of(is_mxfp8, w_scales, w_scale, bias, bias_dtype, out, out_dtype, M, N, K);
  p.x = x;
  p.x_scale = x_scale;
  p.partials = partials;
  p.n_partials = n_partials;
  p.n_vecs = static_cast<int>(M * K / (x_dtype == CK_DTYPE_F32 ? 8 : 16));
  switch (x_dtype) {
    case CK_DTYPE_BF16: return launch<__nv_bfloat16>(is_mxfp8, w, nullptr, p, stream);
    case CK_DTYPE_F16: return launch<__half>(is_mxfp8, w, nullptr, p, stream);
    default: return launch<float>(is_mxfp8, w, nullptr, p, stream);
  }
}

}  // namespace ck
