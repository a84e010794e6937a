// Kernel template and launcher of the block-scaled GEMMs for sm_100a: out[M,N] = cast((A[M,K] . B[N,K]^T) * alpha + bias).
//
//   NVFP4: A, B packed E2M1 (two per byte), E4M3 scale per 16 elements  (kind::mxf4nvf4)
//   MXFP8: A, B E4M3 bytes,                  E8M0 scale per 32 elements  (kind::mxf8f6f4)
//
// One persistent CTA per SM (or, for large problems, one CTA pair per two SMs computing
// 256 x 256 tiles with cta_group::2 instructions), warps with fixed roles:
//   warp 0    TMA producer: per pipeline stage one 128-row x 128-byte box of A, one box of B
//             (128-byte swizzle) and the matching 512-byte scale tiles (linear bulk copies, or
//             3-D tensor maps in a pair) into a STAGES-deep shared-memory ring.
//   warp 1    MMA issuer: per landed stage, copies the stage's scale tiles shared -> tensor
//             memory (tcgen05.cp, up to 12) and issues four tcgen05.mma (32 bytes of K each) into
//             a fp32 accumulator in tensor memory; releases the stage / publishes the accumulator
//             with tcgen05.commit.  The tensor-memory scale columns are buffered per stage like
//             the ring.  (Scale copies on a warp of their own were measured: the extra barrier
//             hop between landing and issue costs 3-15 % at every shape.)
//   warps 2.. epilogue (8 warps; 16 for the fused epilogue, 4 for 64-wide tiles): tcgen05.ld
//             the accumulator into registers, hand it back at once, then alpha * acc + bias,
//             convert, stage the rows in swizzled shared memory and write them with TMA stores
//             while the next tile computes.  The fused variant applies GELU and
//             re-quantizes to NVFP4 instead; the CTAs of a split-K cluster leave raw fp32 partial
//             tiles in shared memory, which the cluster adds; the all-gather variant stores every
//             tile into all ranks' results.
// With NUM_ACC == 2 the epilogue of tile i overlaps the main loop of tile i+1 entirely.
//
// All synchronisation is by mbarriers with bounded waits (ck_sm100.cuh): a protocol error
// raises the device status word instead of hanging.  Kernels are launched with programmatic
// stream serialization; each role waits for the previous kernel (griddepcontrol.wait) only
// before its own first global access.
#pragma once
#include "ck_sm100.cuh"
#include "ck_quant_math.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <vector>

namespace ck {
namespace {

using namespace sm100;

enum class Kind { kNvfp4, kMxfp8 };

constexpr int kTileM = 128;
constexpr int kStageKBytes = 128;   // bytes of K per operand row per stage (one swizzle atom)
constexpr int kMmaKBytes = 32;      // bytes of K per tcgen05.mma
constexpr int kMmaPerStage = kStageKBytes / kMmaKBytes;
// Epilogue warps per CTA: two per 32-lane quarter of tensor memory for the plain epilogue,
// four for the fused one (its activation + quantization arithmetic is ~30 instructions per
// element and must keep up with the tensor pipe), one for a 64-wide tile.
// Timeline builds (-DCK_GEMM_TRACE) keep per-tile stamps in shared memory behind the barriers.
#ifdef CK_GEMM_TRACE
constexpr int kTraceTiles = 40;
constexpr int kTraceSlots = 16;
constexpr int kTraceSmemTiles = 12;
constexpr int kTraceSmemBytes = kTraceSmemTiles * kTraceSlots * 4;
#else
constexpr int kTraceSmemBytes = 0;
#endif

constexpr int epilogue_warps(bool fused, int tile_n) { return (fused && tile_n >= 256) ? 16 : (tile_n <= 64) ? 4 : 8; }
constexpr int num_threads(bool fused, int tile_n) {
  return 64 + 32 * epilogue_warps(fused, tile_n);  // + TMA and MMA warps
}
constexpr int pow2_at_least(int x) { return x <= 32 ? 32 : x <= 64 ? 64 : x <= 128 ? 128 : x <= 256 ? 256 : 512; }

// CTAS == 2: a pair of CTAs (a 2-CTA cluster on neighbouring SMs) computes one 256 x TILE_N
// tile with cta_group::2 instructions.  Each CTA loads its own 128 rows of A and only its
// own half of B's rows, which halves the shared-memory traffic for B - the limiter of the
// single-CTA FP4 kernel.
// OUT_STAGE: the plain epilogue stages the converted tile in shared memory (4 KiB per
// epilogue warp) and writes it with TMA stores.  Storing rows straight from registers puts 32
// partial-line writes per instruction into the SM's memory pipeline, which delays the MMA
// warp's own instructions in that pipeline and starves the tensor cores.
// (OUT_STAGE = number of 4 KiB boxes per epilogue warp, used as a ring; 0 = store from registers.)
template <Kind KIND, int TILE_N, int NUM_ACC, int STAGES, int CTAS, int OUT_STAGE = 0>
struct Config {
  static constexpr int kTileRows = kTileM * CTAS;      // rows of the output tile
  static constexpr int kBRows = TILE_N / CTAS;         // rows of B each CTA loads
  static constexpr int kABytes = kTileM * kStageKBytes;
  static constexpr int kBBytes = kBRows * kStageKBytes;
  // 512-byte scale tiles (128 rows x 4 scale columns) one 128-row block needs per stage:
  // NVFP4 has 16 scale columns per 256 elements, MXFP8 4 per 128 elements.
  static constexpr int kSfTilesPerStage = (KIND == Kind::kNvfp4) ? 4 : 1;
  // 128-row blocks of B's scale tensor a tile can touch (a 192-wide tile straddles two);
  // every CTA needs the scales of all TILE_N columns in its tensor memory.
  static constexpr int kSfbRowBlocks = (TILE_N + 127) / 128;
  static constexpr int kSfaBytes = kSfTilesPerStage * 512;
  static constexpr int kSfbBytes = kSfbRowBlocks * kSfTilesPerStage * 512;
  static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
  static constexpr int kOutStageBytes = OUT_STAGE * epilogue_warps(false, TILE_N) * 4096;
  static constexpr int kRingBytes = (STAGES * kStageBytes + 1023) / 1024 * 1024;
  static constexpr int kSmemBytes = kRingBytes + kOutStageBytes + 3 * TILE_N * 4 /*bias*/ +
                                    1024 /*alignment slack*/ + 256 /*barriers*/ + kTraceSmemBytes;
  // tensor memory columns
  static constexpr int kAccCols = TILE_N;
  static constexpr int kSfaCol = NUM_ACC * kAccCols;
  static constexpr int kSfaColsPerStage = kSfTilesPerStage * 4;
  static constexpr int kSfbCol = kSfaCol + kSfaColsPerStage;  // within one scale buffer
  static constexpr int kSfbColsPerTile = kSfbRowBlocks * 4;
  static constexpr int kSfbColsPerStage = kSfTilesPerStage * kSfbColsPerTile;
  // One set of scale columns per ring stage: the copy of stage s lands in set s, which the
  // stage's "empty" barrier (MMAs retired) frees together with the shared-memory slot.
  static constexpr int kSfColsPerBuf = kSfaColsPerStage + kSfbColsPerStage;
  static_assert(kSfaCol + STAGES * kSfColsPerBuf <= 512, "tensor memory budget exceeded");
  // allocated columns: a power of two; configurations that need at most 256 can share an SM
  static constexpr int kTmemCols = pow2_at_least(kSfaCol + STAGES * kSfColsPerBuf);
  static_assert(CTAS == 1 || CTAS == 2, "one CTA or a CTA pair");
  static_assert(CTAS == 1 || TILE_N % 32 == 0, "a CTA pair needs N % 32 == 0");
  static_assert(TILE_N % 16 == 0 && TILE_N >= 16 && TILE_N <= 256, "invalid MMA N");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget exceeded");
  static constexpr uint32_t kIdesc = make_block_scaled_idesc(KIND == Kind::kNvfp4 ? 1u : 0u,
                                                             KIND == Kind::kNvfp4 ? 0u : 1u, kTileRows, TILE_N);
};

constexpr int kMaxSplits = 8;       // CTAs of a split-K cluster (the portable cluster size)

// Whether and how a tile's K range is split over CTAs.  A kernel of its own for each: code for a split costs the
// calls that do not split 0.1 to 0.6 us (registers, and the tile's index by a division).
enum class Split {
  kNone,
  kCluster,          // the cluster's CTAs add their partial tiles through distributed shared memory
  kOutputs           // CTA s stores its raw fp32 partial tile to destination s
};

struct GemmParams {
  const uint8_t* sfa;      // A scales, tiled layout, [ceil(M/128)][sf_col_tiles] tiles of 512 bytes
  const uint8_t* sfb;      // B scales, same layout over N
  const float* tsa;        // per-tensor scales (device), or null
  const float* tsb;
  const float* alpha;      // overrides tsa*tsb when non-null
  const void* bias;        // [N] or null
  void* out;               // [M, N] row-major
  int bias_dtype;
  int out_dtype;
  int M, N;
  int k_bytes;             // bytes of K per operand row
  int sf_col_tiles;        // 512-byte scale tiles per 128-row block = ceil(K / (4 * block))
  int n_row_blocks_a;      // ceil(M / 128)
  int n_row_blocks_b;      // ceil(N / 128)
  int tiles_m, tiles_n;
  int raster;              // order in which workers walk the tiles: 0 = down the rows first, 1 = along the columns first
  int out_tma;             // the output qualifies for TMA stores (16-byte aligned base and pitch)
  int a_box_rows;          // rows of A in a load: no more than there are
  int n_out;               // destinations of every output tile (1, or one per GPU of an all-gather)
  int splits;              // split-K: CTAs per tile (1 = off); CTA s of a tile covers pipeline stages
  int k_stages_per_split;  //   [s * k_stages_per_split, ...)
  int* status;             // device status word: set non-zero when a wait gave up
  int trace_launch;        // sequence number of the launch (timeline builds only)
  // fused epilogue (FUSED kernels only)
  int activation;          // CK_ACT_*
  uint8_t* rq_codes;       // [M, N/2] NVFP4 codes of the (activated) output, or null
  uint8_t* rq_scales;      // its tiled E4M3 block scales, [roundup(M,128), N/16]
  const float* rq_scale;   // its per-tensor scale (device)
};


// Tile index -> (row block, column block) in the walking order the launch chose.
__device__ __forceinline__ int tile_row_block(const GemmParams& p, int tile) {
  return p.raster == 0 ? tile % p.tiles_m : tile / p.tiles_n;
}
__device__ __forceinline__ int tile_col_block(const GemmParams& p, int tile) {
  return p.raster == 0 ? tile / p.tiles_m : tile % p.tiles_n;
}

// Destinations of the output tile: one tensor map for a plain GEMM; for the column-sharded
// GEMM with a fused all-gather, one per GPU - each a window [M, N_local] at this rank's column
// offset inside that GPU's full [M, N_total] result (peer memory mapped into this process).
constexpr int kMaxOutputs = 8;
struct OutputMaps {
  CUtensorMap m[kMaxOutputs];
};

// Optional per-tile timeline (SM cycle counter) for tuning; compiled in with -DCK_GEMM_TRACE only.
// Per-tile stamps are kept in shared memory (32-bit counts, 12 tiles x 16 slots) and written out
// when the CTA is done: a stamp costs one shared-memory store, so the instrumented kernel behaves
// like the production one (global stores in the loops would queue behind the epilogue's).
// -DCK_GEMM_TRACE_STAGES adds per-stage stamps of the MMA warp, stored to global memory as they
// are taken (these do perturb the kernel).
#ifdef CK_GEMM_TRACE
__device__ long long g_trace[160 * kTraceTiles * kTraceSlots];
__device__ long long g_trace2[160 * 4 * 64];
// per launch (ring of 8) and CTA: global timer (ns) and SM clock at entry, after the dependency wait, at exit
__device__ long long g_trace3[8 * 160 * 8];
__device__ __forceinline__ long long global_timer_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define CK_TRACE3(slot)                                                                              \
  do {                                                                                               \
    if (((slot) == 2 || threadIdx.x == 0) && blockIdx.x < 160) {                                     \
      long long* t3 = g_trace3 + ((p.trace_launch & 7) * 160 + blockIdx.x) * 8 + 2 * (slot);         \
      t3[0] = global_timer_ns();                                                                     \
      t3[1] = clock64();                                                                             \
    }                                                                                                \
  } while (0)
#ifdef CK_GEMM_TRACE_STAGES
#define CK_TRACE2(kind, idx)                                                                         \
  do {                                                                                               \
    if (lane == 0 && (idx) < 64 && blockIdx.x < 160) g_trace2[(blockIdx.x * 4 + (kind)) * 64 + (idx)] = clock64(); \
  } while (0)
#else
#define CK_TRACE2(kind, idx) \
  do {                       \
  } while (0)
#endif
#define CK_TRACE(slot)                                                                               \
  do {                                                                                               \
    if (lane == 0 && tile_it < kTraceSmemTiles) trace_s[tile_it * kTraceSlots + (slot)] = static_cast<uint32_t>(clock64()); \
  } while (0)
#define CK_TRACE_ELECTED(slot)                                                                       \
  do {                                                                                               \
    if (tile_it < kTraceSmemTiles) trace_s[tile_it * kTraceSlots + (slot)] = static_cast<uint32_t>(clock64()); \
  } while (0)
#else
#define CK_TRACE3(slot) \
  do {                  \
  } while (0)
#define CK_TRACE(slot) \
  do {                 \
  } while (0)
#define CK_TRACE2(kind, idx) \
  do {                       \
  } while (0)
#define CK_TRACE_ELECTED(slot) \
  do {                         \
  } while (0)
#endif

// alpha * acc + bias for 32 consecutive output columns of one row.  `bias_s` points at the 32
// fp32 bias values of these columns in shared memory (all lanes read the same addresses).
__device__ __forceinline__ void scale_and_bias(const uint32_t (&raw)[32], float alpha, const float* bias_s,
                                               float (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 b = reinterpret_cast<const float4*>(bias_s)[i];
    v[4 * i + 0] = fmaf(__uint_as_float(raw[4 * i + 0]), alpha, b.x);
    v[4 * i + 1] = fmaf(__uint_as_float(raw[4 * i + 1]), alpha, b.y);
    v[4 * i + 2] = fmaf(__uint_as_float(raw[4 * i + 2]), alpha, b.z);
    v[4 * i + 3] = fmaf(__uint_as_float(raw[4 * i + 3]), alpha, b.w);
  }
}

// Convert and store 32 consecutive output columns of one row.  `vec_ok`: the row pitch and
// column offset allow 32-byte aligned vector stores.
template <typename OutT>
__device__ __forceinline__ void store_row_chunk(OutT* dst, const float (&v)[32], int valid, bool vec_ok) {
  if (valid == 32 && vec_ok) {
    if constexpr (sizeof(OutT) == 2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        Vec256 o;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
            __nv_bfloat162 q = __floats2bfloat162_rn(v[h * 16 + 2 * j], v[h * 16 + 2 * j + 1]);
            o.w[j] = *reinterpret_cast<uint32_t*>(&q);
          } else {
            __half2 q = __floats2half2_rn(v[h * 16 + 2 * j], v[h * 16 + 2 * j + 1]);
            o.w[j] = *reinterpret_cast<uint32_t*>(&q);
          }
        }
        st_global_256_no_allocate(reinterpret_cast<uint8_t*>(dst) + h * 32, o);
      }
    } else {
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        Vec256 o;
#pragma unroll
        for (int j = 0; j < 8; ++j) o.w[j] = __float_as_uint(v[h * 8 + j]);
        st_global_256_no_allocate(reinterpret_cast<uint8_t*>(dst) + h * 32, o);
      }
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (i < valid) {
      if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
        dst[i] = __float2bfloat16_rn(v[i]);
      } else if constexpr (std::is_same<OutT, __half>::value) {
        dst[i] = __float2half_rn(v[i]);
      } else {
        dst[i] = v[i];
      }
    }
  }
}

// Two floats rounded to a 16-bit OutT and packed (first value in the low half), and back.
template <typename OutT>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
    __nv_bfloat162 q = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&q);
  } else {
    __half2 q = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&q);
  }
}
template <typename OutT>
__device__ __forceinline__ void unpack_pair(uint32_t w, float& lo, float& hi) {
  if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
    lo = __uint_as_float(w << 16);
    hi = __uint_as_float(w & 0xFFFF0000u);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    lo = f.x;
    hi = f.y;
  }
}

template <typename OutT>
__device__ __forceinline__ float round_to_out(float x) {
  if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
    return __bfloat162float(__float2bfloat16_rn(x));
  } else if constexpr (std::is_same<OutT, __half>::value) {
    return __half2float(__float2half_rn(x));
  } else {
    return x;
  }
}

// tanh-approximated GELU in fp32: 0.5 x (1 + tanh(u)), u = sqrt(2/pi) (x + 0.044715 x^3),
// evaluated as x * sigmoid(2u) = x / (1 + 2^(-2u log2 e)) with the hardware exp2 and
// reciprocal (relative error ~1e-6, far below the rounding of a 16-bit output type).
__device__ __forceinline__ float gelu_tanh(float x) {
  // x * sigmoid(2u) = x / (1 + 2^(x * (k1 + k2 x^2))), k1 = -2 log2(e) sqrt(2/pi), k2 = 0.044715 k1.
  // The flush-to-zero forms only differ where 1 + 2^(..) exceeds 2^126, i.e. where the exact
  // result is a zero anyway (x below about -10).
  const float w = fmaf(-0.10294324f, x * x, -2.3022082f);
  float t, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(x * w));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + t));
  return x * r;
}

// The same for two values: the multiplies and adds as packed pairs (same roundings, same bits).  The fused
// epilogue was bound by its instruction count (33 per element, 10.4 k cycles a tile against the 6.3 k of its
// main loop); with the pairs here, in the drain and in the quantizer's products it is 21 per element, and fc1 of
// 4608 x 12288 x 3072 takes 99.7 us instead of 108.6 (graph replays), the MLP pair 181.3 instead of 189.9 (eager passes).
__device__ __forceinline__ float2 gelu_tanh_x2(float2 x) {
  const float2 w = fma_x2(make_float2(-0.10294324f, -0.10294324f), mul_x2(x, x), make_float2(-2.3022082f, -2.3022082f));
  const float2 u = mul_x2(x, w);
  float2 t, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t.x) : "f"(u.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t.y) : "f"(u.y));
  t = add_x2(t, make_float2(1.0f, 1.0f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(t.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(t.y));
  return mul_x2(x, r);
}

__device__ __forceinline__ float load_bias(const void* bias, int dtype, int n) {
  if (dtype == CK_DTYPE_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(bias)[n]);
  if (dtype == CK_DTYPE_F16) return __half2float(static_cast<const __half*>(bias)[n]);
  return static_cast<const float*>(bias)[n];
}

// The same in two halves, the load (bits) and the conversion, so that a value can be fetched early: a conversion behind the
// load makes the thread wait for it there.  For the fused epilogue, which has that wait on its critical path; the plain one waits
// for the accumulator anyway and is slower with it (us, value / bits: NVFP4 4096 x 3072 x 3072 19.1 / 19.3, 16384 x 3072 x 1024 37.8 / 38.5).
__device__ __forceinline__ uint32_t load_bias_bits(const void* bias, int dtype, int n) {
  if (dtype == CK_DTYPE_F32) return static_cast<const uint32_t*>(bias)[n];
  return static_cast<const uint16_t*>(bias)[n];
}
__device__ __forceinline__ float bias_of_bits(uint32_t bits, int dtype) {
  if (dtype == CK_DTYPE_BF16) return __uint_as_float(bits << 16);
  if (dtype == CK_DTYPE_F16) return __half2float(__ushort_as_half(static_cast<unsigned short>(bits)));
  return __uint_as_float(bits);
}

template <typename OutT>
__device__ __forceinline__ OutT to_out(float y) {
  if constexpr (std::is_same<OutT, __nv_bfloat16>::value) return __float2bfloat16_rn(y);
  else if constexpr (std::is_same<OutT, __half>::value) return __float2half_rn(y);
  else return y;
}

template <typename OutT>
__device__ __forceinline__ void store_four(OutT* dst, const float (&y)[4]) {
  if constexpr (sizeof(OutT) == 2) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_pair<OutT>(y[0], y[1]), pack_pair<OutT>(y[2], y[3]));
  } else {
    *reinterpret_cast<float4*>(dst) = make_float4(y[0], y[1], y[2], y[3]);
  }
}

__device__ __forceinline__ void sums_scaled(float4 acc, float alpha, const float (&bias)[4], float (&y)[4]) {
  y[0] = fmaf(acc.x, alpha, bias[0]);
  y[1] = fmaf(acc.y, alpha, bias[1]);
  y[2] = fmaf(acc.z, alpha, bias[2]);
  y[3] = fmaf(acc.w, alpha, bias[3]);
}

// Four values at `offset` of every CTA's partial tile, added in split order (all loads before the first add).
__device__ __forceinline__ float4 add_partials(const uint32_t (&base)[kMaxSplits], int splits, uint32_t offset) {
  float4 v[kMaxSplits];
#pragma unroll
  for (int i = 0; i < kMaxSplits; ++i) {
    if (i < splits) v[i] = ld_shared_cluster_f32x4(base[i] + offset);
  }
  float4 acc = v[0];
#pragma unroll
  for (int i = 1; i < kMaxSplits; ++i) {
    if (i < splits) {
      acc.x += v[i].x;
      acc.y += v[i].y;
      acc.z += v[i].z;
      acc.w += v[i].w;
    }
  }
  return acc;
}

// FUSED: the epilogue applies an activation to the output rounded to OutT (what an unfused
// caller would see), optionally stores it, and optionally re-quantizes it to NVFP4 (codes +
// tiled block scales against a static per-tensor scale) as the A operand of the next GEMM.
template <Kind KIND, int TILE_N, int NUM_ACC, int STAGES, int CTAS, typename OutT, bool FUSED, int OUT_STAGE, Split SPLIT = Split::kNone>
__global__ void __launch_bounds__(num_threads(FUSED, TILE_N), 1)
block_scaled_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb,
                         const __grid_constant__ OutputMaps maps_out, const GemmParams p) {
  using Cfg = Config<KIND, TILE_N, NUM_ACC, STAGES, CTAS, OUT_STAGE>;
  static_assert(!(FUSED && OUT_STAGE != 0), "the fused epilogue stores from registers");
  constexpr int kNumEpilogueWarps = epilogue_warps(FUSED, TILE_N);
  constexpr int kThreads = num_threads(FUSED, TILE_N);
  static_assert(TILE_N <= 32 * kNumEpilogueWarps, "one bias value per epilogue thread");
  constexpr bool kCluster = SPLIT == Split::kCluster;
  constexpr bool kOneLane = CTAS == 1, kIssuerLane = CTAS == 1 || FUSED;
  static_assert(SPLIT == Split::kNone || (CTAS == 1 && !FUSED), "only plain one-CTA tiles are split");
  static_assert(SPLIT != Split::kOutputs || (OUT_STAGE != 0 && std::is_same<OutT, float>::value), "raw partial tiles, staged");
  static_assert(!kCluster || kTileM * TILE_N * 4 <= Cfg::kRingBytes, "a partial tile fits in the operand ring");
  // Everything the kernel does until a role's griddepcontrol.wait is independent of the kernel
  // before it in the stream, so the next kernel may be scheduled as early as resources allow.
  pdl_launch_dependents();
  // In a CTA pair, rank 0 (the leader) issues the MMAs and scale copies for both CTAs.
  const uint32_t cta_rank = (CTAS == 2) ? cluster_cta_rank() : 0u;
  const int worker = blockIdx.x / CTAS;        // index of this CTA (pair) among the tile workers
  const int num_workers = gridDim.x / CTAS;
  extern __shared__ uint8_t smem_raw[];
  // operand tiles need 1024-byte alignment for the 128-byte swizzle
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem_a + STAGES * Cfg::kABytes;
  uint8_t* smem_sfa = smem_b + STAGES * Cfg::kBBytes;
  uint8_t* smem_sfb = smem_sfa + STAGES * Cfg::kSfaBytes;
  uint8_t* smem_out = smem + Cfg::kRingBytes;  // 1024-byte aligned (swizzled store boxes)
  float* smem_bias = reinterpret_cast<float*>(smem_out + Cfg::kOutStageBytes);  // [3][TILE_N]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_bias + 3 * TILE_N);
  uint64_t* full_bar = bars;                       // [STAGES] producer -> MMA (operands and scales landed)
  uint64_t* empty_bar = bars + STAGES;             // [STAGES] MMA -> producer (stage and its scale columns free)
  uint64_t* acc_full_bar = bars + 2 * STAGES;      // [NUM_ACC] MMA -> epilogue
  uint64_t* acc_empty_bar = acc_full_bar + NUM_ACC;  // [NUM_ACC] epilogue -> MMA
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(acc_empty_bar + NUM_ACC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
#ifdef CK_GEMM_TRACE
  uint32_t* trace_s = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(bars) + 256);
#endif
  static_assert((2 * STAGES + 2 * NUM_ACC) * 8 + 8 <= 256, "barrier area");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  CK_TRACE3(0);

  // Unsplit one-CTA tiles: ahead of the dependency wait, ask L2 for the first box of B, which is the weight (a prefetch only
  // warms the cache, L2 being the point of coherence).  One: the requests queue in front of the loads in the TMA unit (NVFP4 us, none
  // / one / two / four boxes: 512 x 3072 x 3072 7.58 / 7.47 / 7.53 / 7.56, 128 x 18432 x 3072 9.42 / 9.26 / 9.22 / 9.33, 256 x 3072 x 3072
  // 6.83 / 6.75 / 6.80 / 6.88; split tiles lose, 64 x 3072 x 8192 8.24 / 8.40, and so did pairs).
  if constexpr (CTAS == 1 && SPLIT == Split::kNone) {
    if (warp == 0 && worker < p.tiles_m * p.tiles_n && elect_one()) tma_prefetch_2d(&map_b, 0, tile_col_block(p, worker) * TILE_N);
  }

  // ------------------------------------------------------------------ set-up
  // The producer warp creates the barriers and goes straight to its loads; the other warps
  // meet it at a named barrier it only arrives on (tensor memory is allocated meanwhile).
  // In a pair, every thread arrives on the cluster barrier at once and waits where it first
  // needs the other CTA's barriers to exist.
  uint32_t tmem_base = 0;
  if (warp == 0) {
#ifdef CK_GEMM_TRACE
    for (int i = lane; i < kTraceSmemTiles * kTraceSlots; i += 32) trace_s[i] = 0u;
    __syncwarp();
#endif
    if (lane == 0) {
      *abort_flag = 0;
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(&full_bar[s], 1);
        mbar_init(&empty_bar[s], 1);
      }
      for (int a = 0; a < NUM_ACC; ++a) {
        mbar_init(&acc_full_bar[a], 1);
        mbar_init(&acc_empty_bar[a], kNumEpilogueWarps * CTAS);  // one arrival per epilogue warp (of both CTAs)
      }
      fence_barrier_init();
      prefetch_tensormap(&map_a);
      prefetch_tensormap(&map_b);
      if constexpr (CTAS == 2) {
        prefetch_tensormap(&map_sfa);
        prefetch_tensormap(&map_sfb);
      }
      if constexpr (OUT_STAGE != 0) {
        for (int d = 0; d < p.n_out; ++d) prefetch_tensormap(&maps_out.m[d]);
      }
      __threadfence_block();
    }
    __syncwarp();
    if constexpr (CTAS == 2) {
      cluster_arrive();
      cluster_wait();  // the other CTA's barriers exist before this one's loads report to them
    }
    named_barrier_arrive(2, kThreads);
  } else {
    if constexpr (CTAS == 2) cluster_arrive();
    if (warp == 1) tmem_alloc<CTAS>(tmem_base_slot, Cfg::kTmemCols);
    tc_fence_before_sync();
    named_barrier_sync(2, kThreads);
    if constexpr (CTAS == 2) cluster_wait();
    tc_fence_after_sync();
    tmem_base = *tmem_base_slot;
  }
  CK_TRACE3(1);

  const int num_tiles = p.tiles_m * p.tiles_n;
  const int splits = SPLIT == Split::kNone ? 1 : p.splits;
  // kCluster: what the exchange at the end will scale by and add; the epilogue warps fetch it ahead of their waits
  [[maybe_unused]] float split_alpha = 1.0f;
  [[maybe_unused]] float split_bias[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  const int num_items = num_tiles * splits;
  const int k_stages = (p.k_bytes + kStageKBytes - 1) / kStageKBytes;
  const int total_mma = (p.k_bytes + kMmaKBytes - 1) / kMmaKBytes;

  // Who walks a role's loop.  One CTA: one elected lane all of it.  As whole warps that elect a lane and meet again per stage the
  // issuer took 600 cycles a stage and the producer 480 (128 x 128 tiles; the tensor pipe needs 320 with NVFP4's eight scale copies, 284
  // with MXFP8's two), so, about 400 and 370.  us, whole warps / one lane: NVFP4 64 x 3072 x 3072 6.37 / 5.86, 256 x 3072 x 3072 6.64 / 6.06, 512 x
  // 3072 x 3072 7.36 / 6.85, 256 x 3072 x 12288 13.5 / 13.1, MXFP8 512 x 3072 x 3072 10.8 / 9.8, 128 x 9216 x 3072 10.2 / 9.65.  Pairs are bound by the
  // tensor pipe at 512 cycles, and whole warps serve them better (NVFP4 4096 x 3072 x 3072 18.8 / 19.2, 16384 x 9216 x 3072 180 / 184), except the
  // issuer beside the fused epilogue's sixteen warps (1024 x 12288 x 3072 23.6 / 23.1).  Asking for the next stage's barrier ahead of a stage's MMAs
  // gains nothing.
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (!kOneLane || elect_one()) {
      const uint32_t full_addr = smem_u32(full_bar), empty_addr = smem_u32(empty_bar);
      const uint32_t a_addr = smem_u32(smem_a), b_addr = smem_u32(smem_b), sfa_addr = smem_u32(smem_sfa), sfb_addr = smem_u32(smem_sfb);
      int s = 0;  // ring position and phase as running counters (STAGES is not a power of two)
      uint32_t ph = 0;
      [[maybe_unused]] uint32_t tile_it = 0;
      for (int item = worker; item < num_items; item += num_workers, ++tile_it) {
        const int tile = item / splits;
        const int ks_begin = (item - tile * splits) * p.k_stages_per_split;
        const int ks_end = min(k_stages, ks_begin + p.k_stages_per_split);
        // consecutive workers take neighbouring tiles in the walking order the launch chose (p.raster)
        const int tile_m = tile_row_block(p, tile);
        const int tile_n = tile_col_block(p, tile);
        const int m0 = tile_m * Cfg::kTileRows + static_cast<int>(cta_rank) * kTileM;  // this CTA's rows of A
        const int n0 = tile_n * TILE_N;
        const int b_row = n0 + static_cast<int>(cta_rank) * Cfg::kBRows;
        const int rb_a = m0 / kTileM, rb_b0 = n0 / 128;
        [[maybe_unused]] int rb_b_count = 0;
#pragma unroll
        for (int r = 0; r < Cfg::kSfbRowBlocks; ++r) rb_b_count += (rb_b0 + r < p.n_row_blocks_b) ? 1 : 0;
        // a CTA may own rows past M: it then has no scale row block to load
        [[maybe_unused]] const bool have_sfa = rb_a < p.n_row_blocks_a;
        [[maybe_unused]] const uint8_t* sfa_src = p.sfa + (static_cast<int64_t>(rb_a) * p.sf_col_tiles + ks_begin * Cfg::kSfTilesPerStage) * 512;
        [[maybe_unused]] const uint8_t* sfb_src = p.sfb + (static_cast<int64_t>(rb_b0) * p.sf_col_tiles + ks_begin * Cfg::kSfTilesPerStage) * 512;
        // Operands and scales may come from the kernel before this one.  Its end is waited for only when the first load is all that is
        // left to do: the tile's place, its divisions and the reads of the kernel's arguments took 400 to 800 cycles behind that wait (us,
        // before / so: NVFP4 128 x 1024 x 1024 3.89 / 3.46, 64 x 3072 x 3072 5.86 / 5.45, 512 x 3072 x 3072 6.84 / 6.59, 4096 x 3072 x 3072 18.9 / 18.6).
        bool first = item == worker;
        for (int ks = ks_begin; ks < ks_end; ++ks) {
          mbar_wait(empty_addr + s * 8, ph ^ 1, abort_flag);  // in a pair: signalled from the leader CTA
          if (ks == ks_begin) CK_TRACE_ELECTED(4);
          if (ks == ks_end - 1) CK_TRACE_ELECTED(5);
          if (kOneLane || elect_one()) {
            const uint32_t bar = full_addr + s * 8;
            if constexpr (CTAS == 2) {
              // Every load of both CTAs reports its bytes to the leader's barrier; scale tiles
              // come through 3-D tensor maps {512 B, column tile, row block} so that tiles past
              // the end read as zeros and every stage has the same byte count.
              if (cta_rank == 0) mbar_arrive_expect_tx(bar, 2 * Cfg::kStageBytes);
              if (first) {
                pdl_wait();
                CK_TRACE3(2);
              }
              tma_load_2d_pair(a_addr + s * Cfg::kABytes, &map_a, bar, ks * kStageKBytes, m0);
              tma_load_2d_pair(b_addr + s * Cfg::kBBytes, &map_b, bar, ks * kStageKBytes, b_row);
              tma_load_3d_pair(sfa_addr + s * Cfg::kSfaBytes, &map_sfa, bar, 0, ks * Cfg::kSfTilesPerStage, rb_a);
              tma_load_3d_pair(sfb_addr + s * Cfg::kSfbBytes, &map_sfb, bar, 0, ks * Cfg::kSfTilesPerStage, rb_b0);
            } else {
              const uint32_t sf_bytes = static_cast<uint32_t>(min(Cfg::kSfTilesPerStage, p.sf_col_tiles - ks * Cfg::kSfTilesPerStage)) * 512u;
              mbar_arrive_expect_tx(bar, p.a_box_rows * kStageKBytes + Cfg::kBBytes + sf_bytes * ((have_sfa ? 1 : 0) + rb_b_count));
              if (first) {
                pdl_wait();
                CK_TRACE3(2);
              }
              tma_load_2d(a_addr + s * Cfg::kABytes, &map_a, bar, ks * kStageKBytes, m0);
              tma_load_2d(b_addr + s * Cfg::kBBytes, &map_b, bar, ks * kStageKBytes, b_row);
              if (have_sfa) bulk_load_1d(sfa_addr + s * Cfg::kSfaBytes, sfa_src, sf_bytes, bar);
#pragma unroll
              for (int r = 0; r < Cfg::kSfbRowBlocks; ++r) {
                if (r < rb_b_count) {
                  bulk_load_1d(sfb_addr + s * Cfg::kSfbBytes + r * Cfg::kSfTilesPerStage * 512, sfb_src + static_cast<int64_t>(r) * p.sf_col_tiles * 512,
                               sf_bytes, bar);
                }
              }
              sfa_src += Cfg::kSfTilesPerStage * 512;
              sfb_src += Cfg::kSfTilesPerStage * 512;
            }
          }
          if constexpr (!kOneLane) __syncwarp();
          first = false;
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1 && cta_rank != 0) {
    // second CTA of a pair: the leader issues the MMAs and the scale copies for both
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // Nothing can land before the producer's own dependency wait is over; waiting here too keeps
    // the bounded barrier waits below from running (and giving up) while a long predecessor - a
    // cross-GPU barrier that waits for a late rank, say - is still executing.
    pdl_wait();
    // Descriptors differ between stages only in their start-address field, so the loop
    // carries 32-bit low words; the high words are constants.
    const uint32_t a_lo0 = static_cast<uint32_t>(make_operand_desc_sw128(smem_u32(smem_a)));
    const uint32_t b_lo0 = static_cast<uint32_t>(make_operand_desc_sw128(smem_u32(smem_b)));
    const uint32_t op_hi = static_cast<uint32_t>(make_operand_desc_sw128(0) >> 32);
    const uint32_t sfa_lo0 = static_cast<uint32_t>(make_scale_desc(smem_u32(smem_sfa)));
    const uint32_t sfb_lo0 = static_cast<uint32_t>(make_scale_desc(smem_u32(smem_sfb)));
    const uint32_t sf_hi = static_cast<uint32_t>(make_scale_desc(0) >> 32);
    const uint32_t t_sfa0 = tmem_base + Cfg::kSfaCol;
    const uint32_t t_sfb0 = tmem_base + Cfg::kSfbCol;
    const uint32_t full_addr = smem_u32(full_bar), empty_addr = smem_u32(empty_bar);
    const uint32_t acc_full_addr = smem_u32(acc_full_bar);
    const uint32_t empty_addr_peer = (CTAS == 2) ? map_to_cta(empty_addr, 1) : 0u;
    const uint32_t acc_full_addr_peer = (CTAS == 2) ? map_to_cta(acc_full_addr, 1) : 0u;
    if (!kIssuerLane || elect_one()) {
      [[maybe_unused]] uint32_t it = 0;
      int ring_s = 0;
      uint32_t ring_ph = 0;
      uint32_t tile_it = 0;
      for (int item = worker; item < num_items; item += num_workers, ++tile_it) {
        const int tile = item / splits;
        const int ks_begin = (item - tile * splits) * p.k_stages_per_split;
        const int ks_end = min(k_stages, ks_begin + p.k_stages_per_split);
        const int n0 = tile_col_block(p, tile) * TILE_N;
        const int acc = tile_it % NUM_ACC;
        const uint32_t acc_ph = (tile_it / NUM_ACC) & 1;
        const uint32_t d_tmem = tmem_base + acc * Cfg::kAccCols;
        // B scale words of this tile start (n0 % 128) / 32 columns into the first row block
        const uint32_t sfb_shift = (n0 % 128) / 32;
        for (int ks = ks_begin; ks < ks_end; ++ks, ++it) {
          const int s = ring_s;
          const uint32_t ph = ring_ph;
          if (++ring_s == STAGES) {
            ring_s = 0;
            ring_ph ^= 1u;
          }
          CK_TRACE2(1, it);
          mbar_wait(full_addr + s * 8, ph, abort_flag);
          if (ks == ks_begin) CK_TRACE_ELECTED(2);
          if (ks == ks_end - 1) CK_TRACE_ELECTED(3);
          CK_TRACE2(2, it);
          tc_fence_after_sync();
          if (kIssuerLane || elect_one()) {
            const uint32_t a_lo = a_lo0 + s * (Cfg::kABytes >> 4);
            const uint32_t b_lo = b_lo0 + s * (Cfg::kBBytes >> 4);
            const int n_mma = total_mma - ks * kMmaPerStage;  // left from here on
            const uint32_t t_sfa = t_sfa0 + s * Cfg::kSfColsPerBuf;
            const uint32_t t_sfb_tile = t_sfb0 + s * Cfg::kSfColsPerBuf + sfb_shift;
            // scale tiles of this stage: shared -> tensor memory (512 bytes = 32 descriptor units);
            // the tensor pipe runs them in order ahead of the MMAs that read them
            const uint32_t sfa_lo = sfa_lo0 + s * (Cfg::kSfaBytes >> 4);
            const uint32_t sfb_lo = sfb_lo0 + s * (Cfg::kSfbBytes >> 4);
            const uint32_t t_sfb = t_sfb0 + s * Cfg::kSfColsPerBuf;
#pragma unroll
            for (int t = 0; t < Cfg::kSfTilesPerStage; ++t) {
              tc_copy_scales_32x128b<CTAS>(t_sfa + t * 4, desc64(sfa_lo + t * 32, sf_hi));
#pragma unroll
              for (int r = 0; r < Cfg::kSfbRowBlocks; ++r) {
                tc_copy_scales_32x128b<CTAS>(t_sfb + t * Cfg::kSfbColsPerTile + r * 4,
                                             desc64(sfb_lo + (r * Cfg::kSfTilesPerStage + t) * 32, sf_hi));
              }
            }
            if (ks == ks_begin) {
              // Only now does the tile need its accumulator: the wait for the epilogue to have
              // drained it comes after the first stage has landed.
              CK_TRACE_ELECTED(0);
              mbar_wait(&acc_empty_bar[acc], acc_ph ^ 1, abort_flag);
              CK_TRACE_ELECTED(1);
              tc_fence_after_sync();
            }
            auto mma = [&](int kb) {
              const uint32_t accumulate = (ks != ks_begin || kb != 0) ? 1u : 0u;
              // advancing K inside the swizzle atom = advancing the start address (32 B = 2 units)
              const uint64_t a_desc = desc64(a_lo + kb * 2, op_hi);
              const uint64_t b_desc = desc64(b_lo + kb * 2, op_hi);
              if constexpr (KIND == Kind::kNvfp4) {
                mma_nvfp4<CTAS>(d_tmem, a_desc, b_desc, Cfg::kIdesc, t_sfa + kb * 4, t_sfb_tile + kb * Cfg::kSfbColsPerTile, accumulate);
              } else {
                // one scale tile serves the four MMAs of the stage: byte kb of each scale word
                mma_mxfp8<CTAS>(d_tmem, a_desc, b_desc, idesc_with_scale_ids(Cfg::kIdesc, kb), t_sfa, t_sfb_tile, accumulate);
              }
            };
            if (n_mma >= kMmaPerStage) {
#pragma unroll
              for (int kb = 0; kb < kMmaPerStage; ++kb) mma(kb);
            } else {
              for (int kb = 0; kb < n_mma; ++kb) mma(kb);
            }
            // stage (and its scale columns) reusable once these MMAs retire; in a pair both CTAs are told
            tc_commit<CTAS>(empty_addr + s * 8);
            if constexpr (CTAS == 2) tc_commit<CTAS>(empty_addr_peer + s * 8);
            if (ks == ks_end - 1) {
              tc_commit<CTAS>(acc_full_addr + acc * 8);
              if constexpr (CTAS == 2) tc_commit<CTAS>(acc_full_addr_peer + acc * 8);
            }
          }
          if constexpr (!kIssuerLane) __syncwarp();
          CK_TRACE2(3, it);
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2 ..)
    // Two warps share each 32-lane quarter of tensor memory and split the tile's columns.
    // A warp pulls its whole share of the accumulator into registers with back-to-back
    // tcgen05.ld, hands the accumulator back to the MMA warp at once, and only then does
    // the arithmetic and the stores - so the next tile's main loop overlaps them.
    pdl_wait();  // alpha, bias and the output buffer may belong to the kernel before this one
    const int quarter = warp & 3;  // tensor-memory lanes this warp may read: 32*quarter .. +31
    const int half = (warp - 2) >> 2;  // which share of the tile's columns
    constexpr int kColsPerWarp = TILE_N / (kNumEpilogueWarps / 4);
    constexpr int kChunks = kColsPerWarp / 32;
    static_assert(kColsPerWarp % 32 == 0, "tile width must split into 32-column chunks per warp");
    const int et = threadIdx.x - 64;  // 0 .. 32*kNumEpilogueWarps-1 among the epilogue threads
    float alpha = 1.0f;
    if (p.alpha != nullptr) {
      alpha = ld_f32_dependent(p.alpha);
    } else if (p.tsa != nullptr && p.tsb != nullptr) {
      alpha = ld_f32_dependent(p.tsa) * ld_f32_dependent(p.tsb);
    }
    if constexpr (kCluster) {
      split_alpha = alpha;
      if (p.bias != nullptr) {
        const int tile = worker / splits;
        const int col = tile_col_block(p, tile) * TILE_N + lane * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (col + j < p.N) split_bias[j] = load_bias(p.bias, p.bias_dtype, col + j);
        }
      }
    }
    [[maybe_unused]] float rq_g = 1.0f;
    if constexpr (FUSED) {
      if (p.rq_codes != nullptr) rq_g = ld_f32_dependent(p.rq_scale);
    }
    [[maybe_unused]] const quant::TensorScale rq_ts = quant::make_tensor_scale(rq_g);
    OutT* out = static_cast<OutT*>(p.out);
    const bool vec_ok = (static_cast<int64_t>(p.N) * sizeof(OutT)) % 32 == 0 &&
                        (reinterpret_cast<uintptr_t>(p.out) & 31u) == 0 && (TILE_N * sizeof(OutT)) % 32 == 0;
    const uint32_t acc_empty_leader = (CTAS == 2) ? map_to_cta(smem_u32(acc_empty_bar), 0) : 0u;
    // The fused 16-bit epilogue never holds the raw accumulator: it drains 16 columns at a
    // time and keeps alpha * acc + bias rounded to OutT as packed pairs (a quarter of the
    // registers); the others pull their whole share with back-to-back loads.
    constexpr bool kPackedDrain = FUSED && sizeof(OutT) == 2;
    constexpr bool kWarpBias = kPackedDrain;  // each warp its own columns' bias (below)
    constexpr int kBiasPerThread = kWarpBias ? kColsPerWarp / 32 : 1;
    const int bias_col = kWarpBias ? half * kColsPerWarp + lane : et;
    [[maybe_unused]] uint32_t out_box = 0;  // boxes this warp has staged so far (ring index)
    uint32_t tile_it = 0;
    for (int item = worker; item < num_items; item += num_workers, ++tile_it) {
      const int tile = item / splits;
      const int tile_m = tile_row_block(p, tile);
      const int tile_n = tile_col_block(p, tile);
      const int row = tile_m * Cfg::kTileRows + static_cast<int>(cta_rank) * kTileM + quarter * 32 + lane;
      const int n0 = tile_n * TILE_N;
      const int acc = tile_it % NUM_ACC;
      const uint32_t acc_ph = (tile_it / NUM_ACC) & 1;
      // Bias of a tile's columns as fp32 in shared memory, three buffers in rotation: the buffer of tile t is filled
      // while tile t - 1 is in its epilogue, right after the drain, with values fetched ahead of the wait for the
      // accumulator, whose latency that wait hides.
      // Plain tiles and fp32: every thread fetches one value, and the warps meet at a barrier after the drain, where they
      // are aligned anyway; a warp then runs at most one tile ahead of the slowest, hence the third buffer.
      // Fused 16-bit tiles: every warp fetches the columns it reads itself (the four warps of the same columns write the same
      // values; tile t + 3's come behind the accumulator of t + 2, which waits for all warps' drains of t, where the bias of t
      // is read), since a barrier a tile made each of sixteen warps wait for the one with the longest chains: us, barrier / so,
      // bf16 4608 x 8192 x 2048 47.7 / 44.8, 4608 x 12288 x 3072 80.1 / 77.6 (under the power limit 93.9 / 91.5), fp16 81.1 / 78.9; one tile to
      // a worker, 128 x 12288 x 3072, 8.95 / 8.98.  With fp32 it lost (77.6 / 78.3), and so did plain pairs (36864 x 9216 x 3072 407 / 416).
      float* bias_s = smem_bias + (tile_it % 3) * TILE_N;
      const bool with_bias = p.bias != nullptr;
      if (tile_it == 0) {
        if constexpr (kWarpBias) {
          // all fetched before the first is converted: one after the other, their latencies stood in front of a short main loop
          // (us, 128 x 12288 x 256 fp16 5.60 / 5.49, 16 x 2496 x 256 5.25 / 5.10)
          uint32_t bits[kBiasPerThread];
#pragma unroll
          for (int i = 0; i < kBiasPerThread; ++i) {
            const int n = n0 + bias_col + 32 * i;
            bits[i] = (with_bias && n < p.N) ? load_bias_bits(p.bias, p.bias_dtype, n) : 0u;
          }
#pragma unroll
          for (int i = 0; i < kBiasPerThread; ++i) bias_s[bias_col + 32 * i] = bias_of_bits(bits[i], p.bias_dtype);
          __syncwarp();
        } else {
          if (et < TILE_N) bias_s[et] = (with_bias && n0 + et < p.N) ? load_bias(p.bias, p.bias_dtype, n0 + et) : 0.0f;
          asm volatile("bar.sync 1, %0;" ::"n"(32 * kNumEpilogueWarps) : "memory");  // epilogue warps only
        }
      }
      const int next_item = item + num_workers;
      const bool has_next = next_item < num_items;
      std::conditional_t<FUSED, uint32_t, float> bias_prefetched[kBiasPerThread] = {};  // bits or value: zero is 0.0 in every type
      if (has_next && (kWarpBias || et < TILE_N)) {
#pragma unroll
        for (int i = 0; i < kBiasPerThread; ++i) {
          const int n = tile_col_block(p, next_item / splits) * TILE_N + bias_col + 32 * i;
          if (with_bias && n < p.N) {
            if constexpr (FUSED) bias_prefetched[i] = load_bias_bits(p.bias, p.bias_dtype, n);
            else bias_prefetched[i] = load_bias(p.bias, p.bias_dtype, n);
          }
        }
      }
      if (warp == 2) CK_TRACE(6);
      mbar_wait(&acc_full_bar[acc], acc_ph, abort_flag);  // in a pair: committed from the leader CTA
      if (warp == 2) CK_TRACE(7);
      // the aligned loads below want the whole warp, of which the last tile's epilogue may have sent the rows past M another way
      if constexpr (FUSED) __syncwarp();
      tc_fence_after_sync();
      const int c0 = half * kColsPerWarp;
      const uint32_t t_row = tmem_base + acc * Cfg::kAccCols + (static_cast<uint32_t>(quarter * 32) << 16) + c0;
      [[maybe_unused]] uint32_t buf[kPackedDrain ? 1 : kChunks][32];
      [[maybe_unused]] uint32_t pk[kPackedDrain ? kChunks : 1][16];
      if constexpr (kPackedDrain) {
        // 16 columns at a time, the next ones on their way while these are scaled: the tensor pipe idles until the drain ends.
        // 32 at a time and one after the other / so, us: bf16 4608 x 12288 x 3072 80.5 / 79.9, 1024 x 12288 x 3072 23.8 / 23.6, fp16 4608 x
        // 12288 x 3072 87.2 / 81.7, 1000 x 8192 x 2048 16.2 / 15.7.
        uint32_t part[2][16];
        tmem_load_32x16(t_row, part[0]);
#pragma unroll
        for (int h = 0; h < 2 * kChunks; ++h) {
          tmem_load_wait();
          if (h + 1 < 2 * kChunks) tmem_load_32x16(t_row + (h + 1) * 16, part[(h + 1) % 2]);
          const float2* b2 = reinterpret_cast<const float2*>(bias_s + c0 + h * 16);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float2 y = fma_x2(make_float2(__uint_as_float(part[h % 2][2 * i]), __uint_as_float(part[h % 2][2 * i + 1])),
                                    make_float2(alpha, alpha), b2[i]);
            pk[h / 2][8 * (h % 2) + i] = pack_pair<OutT>(y.x, y.y);
          }
        }
      } else {
#pragma unroll
        for (int c = 0; c < kChunks; ++c) tmem_load_32x32(t_row + c * 32, buf[c]);
        tmem_load_wait();
      }
      if (warp == 2) CK_TRACE(8);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if constexpr (CTAS == 2) {
          mbar_arrive_cluster(acc_empty_leader + acc * 8);  // the leader's barrier counts both CTAs' warps
        } else {
          mbar_arrive(&acc_empty_bar[acc]);
        }
      }
      if constexpr (kCluster) {
        // Raw partial to the CTA's own shared memory: row r at r * TILE_N * 4 bytes, its 16-byte unit u
        // at position u ^ (r % 8) (the eight rows of a store phase meet eight different bank groups).
        const int r = quarter * 32 + lane;
        const uint32_t part_row = smem_u32(smem) + r * (TILE_N * 4);
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int u = (c0 + c * 32) / 4 + j;
            st_shared_128(part_row + ((u ^ (r & 7)) << 4), buf[c][4 * j], buf[c][4 * j + 1], buf[c][4 * j + 2], buf[c][4 * j + 3]);
          }
        }
        continue;
      }
      if (has_next) {
        if (kWarpBias || et < TILE_N) {
#pragma unroll
          for (int i = 0; i < kBiasPerThread; ++i) {
            float b;
            if constexpr (FUSED) b = bias_of_bits(bias_prefetched[i], p.bias_dtype);
            else b = bias_prefetched[i];
            smem_bias[((tile_it + 1) % 3) * TILE_N + bias_col + 32 * i] = b;
          }
        }
        if constexpr (kWarpBias) {
          __syncwarp();
        } else {
          asm volatile("bar.sync 1, %0;" ::"n"(32 * kNumEpilogueWarps) : "memory");  // epilogue warps only
        }
      }
      OutT* out_row = out + static_cast<int64_t>(row) * p.N + n0 + c0;
      if constexpr (!FUSED) {
        bool staged = false;
        if constexpr (OUT_STAGE != 0) staged = p.out_tma != 0;
        if (staged) {
          if constexpr (OUT_STAGE != 0) {
            // The warp's 32 rows x 128 bytes of converted output go to its staging box in the
            // 128-byte-swizzled layout (16-byte unit j of row r at r*128 + ((j ^ r%8) * 16):
            // conflict-free for the 8 lanes of a store phase), then one TMA store writes whole
            // lines; rows past M and columns past N are clipped by the tensor map.
            constexpr int kBoxCols = 128 / static_cast<int>(sizeof(OutT));
            constexpr int kChunksPerBox = kBoxCols / 32;          // 2 for 16-bit outputs, 1 for fp32
            constexpr int kUnitsPerChunk = 32 * static_cast<int>(sizeof(OutT)) / 16;
            static_assert((kChunks / kChunksPerBox - 1) * kNumEpilogueWarps * 4096 <= Cfg::kRingBytes,
                          "the last tile's extra store boxes fit in the idle operand ring");
            const uint32_t stage_warp = smem_u32(smem_out) + (warp - 2) * (OUT_STAGE * 4096);
            const int row0 = tile_m * Cfg::kTileRows + static_cast<int>(cta_rank) * kTileM + quarter * 32;
#pragma unroll
            for (int c = 0; c < kChunks; ++c) {
              // A CTA's last tile finds the operand ring idle (every load has landed and every
              // MMA has retired before its accumulator was published): its second and later
              // boxes are staged there, so the warp never waits for a store to release a box.
              const bool in_ring = !has_next && c >= kChunksPerBox;
              const uint32_t stage_box =
                  in_ring ? smem_u32(smem) + ((c / kChunksPerBox - 1) * kNumEpilogueWarps + (warp - 2)) * 4096
                          : stage_warp + (out_box % OUT_STAGE) * 4096;
              const uint32_t stage_row = stage_box + lane * 128;
              if (c == 0 && warp == 2) CK_TRACE(10);
              if (c % kChunksPerBox == 0 && !in_ring) {
                if (lane == 0) bulk_wait_group_read<OUT_STAGE - 1>();  // the store that last used this box has read it
                __syncwarp();
              }
              if (c == 0 && warp == 2) CK_TRACE(11);
              if (c == 2 && warp == 2) CK_TRACE(14);
              float v[32];
              scale_and_bias(buf[c], alpha, bias_s + c0 + c * 32, v);
#pragma unroll
              for (int u = 0; u < kUnitsPerChunk; ++u) {
                uint32_t w[4];
                if constexpr (sizeof(OutT) == 2) {
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
                      __nv_bfloat162 q = __floats2bfloat162_rn(v[u * 8 + 2 * j], v[u * 8 + 2 * j + 1]);
                      w[j] = *reinterpret_cast<uint32_t*>(&q);
                    } else {
                      __half2 q = __floats2half2_rn(v[u * 8 + 2 * j], v[u * 8 + 2 * j + 1]);
                      w[j] = *reinterpret_cast<uint32_t*>(&q);
                    }
                  }
                } else {
#pragma unroll
                  for (int j = 0; j < 4; ++j) w[j] = __float_as_uint(v[u * 4 + j]);
                }
                const int unit = (c % kChunksPerBox) * kUnitsPerChunk + u;
                st_shared_128(stage_row + (((unit ^ lane) & 7) << 4), w[0], w[1], w[2], w[3]);
              }
              if (c == 0 && warp == 2) CK_TRACE(12);
              if (c == 1 && warp == 2) CK_TRACE(13);
              if (c % kChunksPerBox == kChunksPerBox - 1) {
                fence_proxy_async();  // the staged bytes become visible to the TMA engine
                __syncwarp();
                const int col = n0 + c0 + (c / kChunksPerBox) * kBoxCols;
                if (lane == 0 && row0 < p.M && col < p.N) {
                  if constexpr (SPLIT == Split::kOutputs) {
                    tma_store_2d_addr(&maps_out.m[item - tile * splits], stage_box, col, row0);  // this item's partial
                  } else {
                    // the same staged box goes to every destination (peer stores cross NVLink)
                    for (int d = 0; d < p.n_out; ++d) tma_store_2d_addr(&maps_out.m[d], stage_box, col, row0);
                  }
                }
                // (an empty group when nothing was stored keeps the ring's group count in step)
                if (lane == 0) bulk_commit_group();
                if (c == 1 && warp == 2) CK_TRACE(15);
                if (!in_ring) ++out_box;
              }
            }
          }
        } else {
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            const int valid = min(32, p.N - (n0 + c0 + c * 32));
            if (row < p.M && valid > 0) {
              float v[32];
              scale_and_bias(buf[c], alpha, bias_s + c0 + c * 32, v);
              store_row_chunk<OutT>(out_row + c * 32, v, valid, vec_ok);
            }
          }
        }
      } else {
        // Re-quantization needs whole 64-column groups (4 scale columns = one 32-bit word of
        // the tiled scale layout); the host guarantees N % 64 == 0 when it is requested.
        static_assert(kChunks % 2 == 0, "fused epilogue works on pairs of 32-column chunks");  // 64-column groups
        const int rq_col_tiles = (p.N / 16 + 3) / 4;
        const int rows_pad = (p.M + 127) / 128 * 128;
        uint32_t scale_word = 0;
        if constexpr (kPackedDrain) {
          // The values an unfused caller would see are the accumulators rounded to OutT: the
          // activation works on the packed pairs, and the re-quantization runs on the packed
          // words exactly as the stand-alone quantizer does.
          // GELU and re-quantization alone of a row's whole share of columns, the usual call: two blocks at a time in one
          // straight piece of code, in which their serial chains and the activation's overlap.  A tile took its epilogue 9.2 k
          // cycles (1.5 k more waiting for the next tile's bias behind its conversion) beside a main loop of 6.5 k.  fc1 in graph
          // replays, before / one / two / four blocks at a time: 4608 x 12288 x 3072 85.4 / 85.6 / 81.5 / 89.7 us (four spill; with the drain and the
          // blocks' arithmetic as they are now two take 79.9, one at a time beside the next one's GELU 81.1 to 83.8), 16384 x 8192
          // x 2048 175.8 / 166.9 / 158.7 / 180.2.
          if (p.activation == CK_ACT_GELU_TANH && p.out == nullptr && row < p.M && n0 + c0 + kColsPerWarp <= p.N) {
#pragma unroll
            for (int c = 0; c < kChunks; c += 2) {
              const int col = n0 + c0 + c * 32;
              uint32_t codes[4][2], sb[4];
#pragma unroll
              for (int h = 0; h < 4; h += 2) {
                quant::Sixteen<OutT> x16[2];
                uint32_t c2[2][2], s2[2];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  float2 x;
                  unpack_pair<OutT>(pk[c + (8 * h + i) / 16][(8 * h + i) % 16], x.x, x.y);
                  x = gelu_tanh_x2(x);
                  x16[i / 8].w[i % 8] = pack_pair<OutT>(x.x, x.y);
                }
                quant::nvfp4_blocks<OutT, true, 2, false>(x16, rq_ts, c2, s2);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  codes[h + i][0] = c2[i][0];
                  codes[h + i][1] = c2[i][1];
                  sb[h + i] = s2[i];
                }
              }
              uint4* const dst = reinterpret_cast<uint4*>(p.rq_codes + static_cast<int64_t>(row) * (p.N >> 1) + (col >> 1));
              dst[0] = make_uint4(codes[0][0], codes[0][1], codes[1][0], codes[1][1]);
              dst[1] = make_uint4(codes[2][0], codes[2][1], codes[3][0], codes[3][1]);
              *reinterpret_cast<uint32_t*>(p.rq_scales + swizzled_scale_offset(row, col >> 4, rq_col_tiles)) =
                  sb[0] | (sb[1] << 8) | (sb[2] << 16) | (sb[3] << 24);
            }
            if (warp == 2) CK_TRACE(9);
            continue;
          }
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            const int col = n0 + c0 + c * 32;
            const int valid = min(32, p.N - col);
            if (valid <= 0) continue;
            if (row < p.M) {
              if (p.activation == CK_ACT_GELU_TANH) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  float2 x;
                  unpack_pair<OutT>(pk[c][i], x.x, x.y);
                  x = gelu_tanh_x2(x);
                  pk[c][i] = pack_pair<OutT>(x.x, x.y);
                }
              }
              if (p.out != nullptr) {
                if (vec_ok && valid == 32) {
                  Vec256 o0, o1;
#pragma unroll
                  for (int i = 0; i < 8; ++i) {
                    o0.w[i] = pk[c][i];
                    o1.w[i] = pk[c][8 + i];
                  }
                  st_global_256_no_allocate(out_row + c * 32, o0);
                  st_global_256_no_allocate(out_row + c * 32 + 16, o1);
                } else {
#pragma unroll
                  for (int i = 0; i < 16; ++i) {  // N % 8 == 0: pairs never straddle the edge
                    if (2 * i < valid) *reinterpret_cast<uint32_t*>(out_row + c * 32 + 2 * i) = pk[c][i];
                  }
                }
              }
            }
            if (p.rq_codes != nullptr) {  // N % 64 == 0 here: every chunk is whole
              if (row < p.M) {
                // out of line: inlined here its registers cost the straight code above 4 % (81.5 us against 87.0 at 4608 x 12288 x 3072)
                const quant::BlockCodes lo = quant::nvfp4_block_packed_call<OutT, true>(pk[c][0], pk[c][1], pk[c][2], pk[c][3], pk[c][4], pk[c][5],
                                                                                        pk[c][6], pk[c][7], rq_ts);
                const quant::BlockCodes hi = quant::nvfp4_block_packed_call<OutT, true>(pk[c][8], pk[c][9], pk[c][10], pk[c][11], pk[c][12],
                                                                                        pk[c][13], pk[c][14], pk[c][15], rq_ts);
                *reinterpret_cast<uint4*>(p.rq_codes + static_cast<int64_t>(row) * (p.N >> 1) + (col >> 1)) =
                    make_uint4(lo.lo, lo.hi, hi.lo, hi.hi);
                scale_word |= (lo.scale_byte | (hi.scale_byte << 8)) << (16 * (c & 1));
              }
              if ((c & 1) && row < rows_pad) {
                // rows between M and the next multiple of 128 are padding of the scale tensor: zero
                // this chunk and the previous one cover scale columns (col/16 - 2) .. (col/16 + 1)
                const int64_t off = swizzled_scale_offset(row, (col >> 4) - 2, rq_col_tiles);
                *reinterpret_cast<uint32_t*>(p.rq_scales + off) = scale_word;
                scale_word = 0;
              }
            }
          }
        } else {
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            const int col = n0 + c0 + c * 32;
            const int valid = min(32, p.N - col);
            if (valid <= 0) continue;
            float v[32];
            if (row < p.M) {
              scale_and_bias(buf[c], alpha, bias_s + c0 + c * 32, v);
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                float y = round_to_out<OutT>(v[i]);
                if (p.activation == CK_ACT_GELU_TANH) y = round_to_out<OutT>(gelu_tanh(y));
                v[i] = y;
              }
              if (p.out != nullptr) store_row_chunk<OutT>(out_row + c * 32, v, valid, vec_ok);
            }
            if (p.rq_codes != nullptr) {
              if (row < p.M) {
                float lo16[16], hi16[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  lo16[i] = v[i];
                  hi16[i] = v[16 + i];
                }
                uint32_t w0, w1, w2, w3, s0, s1;
                quant::nvfp4_block<true>(lo16, rq_g, true, w0, w1, s0);
                quant::nvfp4_block<true>(hi16, rq_g, true, w2, w3, s1);
                *reinterpret_cast<uint4*>(p.rq_codes + static_cast<int64_t>(row) * (p.N >> 1) + (col >> 1)) =
                    make_uint4(w0, w1, w2, w3);
                scale_word |= (s0 | (s1 << 8)) << (16 * (c & 1));
              }
              if ((c & 1) && row < rows_pad) {
                const int64_t off = swizzled_scale_offset(row, (col >> 4) - 2, rq_col_tiles);
                *reinterpret_cast<uint32_t*>(p.rq_scales + off) = scale_word;
                scale_word = 0;
              }
            }
          }
        }
      }
      if (warp == 2) CK_TRACE(9);
    }
    if constexpr (OUT_STAGE != 0) {
      // shared memory stays valid until the last store has read it; stores to other GPUs are
      // waited for to the end, so that they precede whatever follows this kernel on the stream
      if (lane == 0) {
        if (p.n_out > 1) {
          bulk_wait_group0();
        } else {
          bulk_wait_group_read0();
        }
      }
    }
  }

  // ------------------------------------------------------------------ split-K: the cluster adds its partial tiles
  // Every CTA of the cluster ran one item (the host launches tiles * splits CTAs); its partial lies in
  // its own operand ring, which is idle: all loads have landed and all MMAs have retired before the
  // accumulator was published.  Each CTA reads its share of the tile from all of them over distributed
  // shared memory and adds in split order, so the result does not depend on scheduling; no workspace,
  // no second kernel, no counters to keep zero - and so the one-call linears split as well.  Measured
  // against partial tiles through L2 (graph replays, us; linear = quantize + GEMM in one call, which
  // had no workspace and ran unsplit): MXFP8 1 x 3072 x 12288 linear 30.1 -> 12.5, 256 rows 33.0 -> 24.4;
  // NVFP4 1 x 1024 x 15360 GEMM 8.7 -> 6.3, linear 21.8 -> 8.1; 64 x 3072 x 12288 11.3 -> 9.6.  A cluster
  // must find its SMs in one part of the chip: where that costs too many CTAs per tile, the GEMMs that have
  // a workspace go through it (choose_splits in ck_gemm.cu).
  if constexpr (kCluster) {
    __syncwarp();
    cluster_sync_all();
    if (warp >= 2) {
      const int rank = static_cast<int>(cluster_cta_rank());
      const int tile = worker / splits;
      const uint32_t part = smem_u32(smem);
      uint32_t base[kMaxSplits];
#pragma unroll
      for (int i = 0; i < kMaxSplits; ++i) base[i] = map_to_cta(part, i < splits ? i : 0);
      // a warp takes one row of the tile, a lane four neighbouring columns
      const int row0 = tile_row_block(p, tile) * kTileM;
      const int col = tile_col_block(p, tile) * TILE_N + lane * 4;
      const bool in_cols = col < p.N;  // N % 8 == 0: a group of four never straddles the edge
      const int rows = min(kTileM, p.M - row0);
      for (int r = rank + splits * (warp - 2); r < rows; r += splits * kNumEpilogueWarps) {
        const float4 acc = add_partials(base, splits, r * (TILE_N * 4) + ((lane ^ (r & 7)) << 4));
        float y[4];
        sums_scaled(acc, split_alpha, split_bias, y);
        if (in_cols) store_four(static_cast<OutT*>(p.out) + static_cast<int64_t>(row0 + r) * p.N + col, y);
      }
    }
    __syncwarp();
    cluster_sync_all();  // no CTA leaves while another may still read its partial
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  CK_TRACE3(3);
#ifdef CK_GEMM_TRACE
  if (blockIdx.x < 160) {
    for (int i = threadIdx.x; i < kTraceSmemTiles * kTraceSlots; i += blockDim.x) {
      g_trace[(blockIdx.x * kTraceTiles + i / kTraceSlots) * kTraceSlots + i % kTraceSlots] = trace_s[i];
    }
  }
#endif
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicExch(p.status, 1);
    // give copies that may still be in flight time to land before the CTA's memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if constexpr (CTAS == 2) cluster_sync_all();  // no CTA leaves while its partner may still signal it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<CTAS>(tmem_base, Cfg::kTmemCols);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
  });
  return fn;
}

// Tensor maps are a pure function of (address, extents, box): a small per-thread table keeps the
// ones of recent calls, so that a layer called again with the same buffers pays no encode.
struct MapKey {
  int tag;
  const void* base;
  int64_t d0, d1, d2, d3;
  bool operator==(const MapKey& o) const {
    return tag == o.tag && base == o.base && d0 == o.d0 && d1 == o.d1 && d2 == o.d2 && d3 == o.d3;
  }
};

template <typename Encode>
int cached_map(CUtensorMap* map, const MapKey& key, Encode&& encode) {
  struct Entry {
    MapKey key;
    CUtensorMap map;
    bool valid;
  };
  constexpr int kEntries = 128;
  thread_local std::vector<Entry> table(kEntries);  // on the heap: keeps the library's TLS block small
  uint64_t h = reinterpret_cast<uintptr_t>(key.base) >> 8;
  h = (h ^ (h >> 17) ^ static_cast<uint64_t>(key.tag) * 0x9E3779B97F4A7C15ull ^ static_cast<uint64_t>(key.d1) * 0xC2B2AE3D27D4EB4Full);
  Entry& e = table[(h ^ (h >> 29)) % kEntries];
  if (e.valid && e.key == key) {
    *map = e.map;
    return CK_OK;
  }
  if (int rc = encode(map)) return rc;
  e.key = key;
  e.map = *map;
  e.valid = true;
  return CK_OK;
}

// Row-major [rows, row_bytes] byte matrix, boxes of 128 bytes x box_rows rows, 128-byte swizzle.
int encode_operand_map(CUtensorMap* map, const void* base, int64_t rows, int64_t row_bytes, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return fail(CK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kStageKBytes), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box,
                        elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(CK_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", static_cast<int>(r));
  return CK_OK;
}

// Scale tensor in the tiled layout as a 3-D array {128 x uint32 (one 512-byte tile), column
// tile, row block}; a box is `tiles` consecutive column tiles of `box_row_blocks` row blocks.
int encode_scale_map(CUtensorMap* map, const void* base, int64_t row_blocks, int64_t col_tiles, int tiles, int box_row_blocks) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return fail(CK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t dims[3] = {128, static_cast<cuuint64_t>(col_tiles), static_cast<cuuint64_t>(row_blocks)};
  const cuuint64_t strides[2] = {512, static_cast<cuuint64_t>(col_tiles) * 512};
  const cuuint32_t box[3] = {128, static_cast<cuuint32_t>(tiles), static_cast<cuuint32_t>(box_row_blocks)};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void*>(base), dims, strides, box,
                        elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(CK_ERR_CUDA, "cuTensorMapEncodeTiled (scales) failed with code %d", static_cast<int>(r));
  return CK_OK;
}

// Row-major [rows, cols] output of `elem_bytes`-wide elements: boxes of 32 rows x 128 bytes,
// 128-byte swizzle (the layout the epilogue stages its rows in).
int encode_output_map(CUtensorMap* map, void* base, int64_t rows, int64_t cols, int elem_bytes, int64_t pitch_elems) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return fail(CK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const CUtensorMapDataType type = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch_elems) * elem_bytes};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem_bytes), 32};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r = fn(map, type, 2, base, dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(CK_ERR_CUDA, "cuTensorMapEncodeTiled (output) failed with code %d", static_cast<int>(r));
  return CK_OK;
}

int make_operand_map(CUtensorMap* map, const void* base, int64_t rows, int64_t row_bytes, int box_rows) {
  return cached_map(map, MapKey{0, base, rows, row_bytes, box_rows, 0},
                    [&](CUtensorMap* m) { return encode_operand_map(m, base, rows, row_bytes, box_rows); });
}

int make_scale_map(CUtensorMap* map, const void* base, int64_t row_blocks, int64_t col_tiles, int tiles, int box_row_blocks) {
  return cached_map(map, MapKey{1, base, row_blocks, col_tiles, tiles, box_row_blocks},
                    [&](CUtensorMap* m) { return encode_scale_map(m, base, row_blocks, col_tiles, tiles, box_row_blocks); });
}

int make_output_map(CUtensorMap* map, void* base, int64_t rows, int64_t cols, int elem_bytes, int64_t pitch_elems) {
  return cached_map(map, MapKey{2, base, rows, cols, elem_bytes, pitch_elems},
                    [&](CUtensorMap* m) { return encode_output_map(m, base, rows, cols, elem_bytes, pitch_elems); });
}

// Where the output goes (host side): `n` buffers (1 = plain GEMM), each holding this GEMM's
// [M, N] block at column `col_offset` of a row-major matrix with `pitch` columns.
struct OutputSpec {
  void* const* ptrs = nullptr;
  int n = 1;
  int64_t pitch = 0;
  int64_t col_offset = 0;
  bool plain(int64_t N) const { return n == 1 && pitch == N && col_offset == 0; }
};

// The two operand matrices (device pointers): A [M, k_bytes], B [N, k_bytes] row-major bytes.
struct Operands {
  const void* a;
  const void* b;
};

// Clusters of `splits` CTAs of this configuration that can run at once on the current device, one CTA to an SM.
template <Kind KIND, int TILE_N, int NUM_ACC, int STAGES, typename OutT, int OUT_STAGE>
int split_clusters(int splits, int* out) {
  using Cfg = Config<KIND, TILE_N, NUM_ACC, STAGES, 1, OUT_STAGE>;
  static std::atomic<int> cached[64][kMaxSplits + 1];
  int dev = 0;
  CK_CUDA(cudaGetDevice(&dev));
  int n = (dev >= 0 && dev < 64) ? cached[dev][splits].load(std::memory_order_relaxed) : 0;
  if (n == 0) {
    auto kernel = block_scaled_gemm_kernel<KIND, TILE_N, NUM_ACC, STAGES, 1, OutT, false, OUT_STAGE, Split::kCluster>;
    CK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(num_threads(false, TILE_N));
    cfg.gridDim = dim3(static_cast<unsigned>(sm_count() / splits * splits));
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
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

template <Kind KIND, int TILE_N, int NUM_ACC, int STAGES, int CTAS, typename OutT, bool FUSED, int OUT_STAGE = 0, Split SPLIT = Split::kNone>
int launch_config(const Operands& ops, GemmParams p, const OutputSpec& os, cudaStream_t stream) {
  using Cfg = Config<KIND, TILE_N, NUM_ACC, STAGES, CTAS, OUT_STAGE>;
  auto kernel = block_scaled_gemm_kernel<KIND, TILE_N, NUM_ACC, STAGES, CTAS, OutT, FUSED, OUT_STAGE, SPLIT>;
  // only the tensor maps this configuration uses are encoded (host time is visible for small problems)
  CUtensorMap map_a, map_b;
  // No rows past M in a box where one row block has them all: filling them made a load of a small activation, less than 128 KiB, slow (us,
  // boxes of 128 rows / of M: NVFP4 33 x 12288 x 6144 15.2 / 10.9, 33 x 9216 x 3072 7.1 / 6.4, MXFP8 33 x 9216 x 3072 11.3 / 9.5, 33 x 3072 x 3072 7.1 / 6.5;
  // 96 x 9216 x 3072 6.5 / 6.5).  What the slot then holds of an earlier stage goes to rows of the accumulator that are not stored.
  p.a_box_rows = CTAS == 1 && p.M < kTileM ? p.M : kTileM;
  if (int rc = make_operand_map(&map_a, ops.a, p.M, p.k_bytes, p.a_box_rows)) return rc;
  if (int rc = make_operand_map(&map_b, ops.b, p.N, p.k_bytes, Cfg::kBRows)) return rc;
  // the dynamic shared-memory opt-in is per device: do it once for each device that launches
  static std::atomic<bool> configured[64];
  int dev = 0;
  CK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    CK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  p.tiles_m = static_cast<int>(ceil_div(p.M, Cfg::kTileRows));
  p.tiles_n = static_cast<int>(ceil_div(p.N, TILE_N));
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(num_threads(FUSED, TILE_N));
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  constexpr bool cluster_split = SPLIT == Split::kCluster;
  attr[0].val.clusterDim.x = cluster_split ? p.splits : CTAS;  // split-K: the CTAs of one tile are a cluster
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  // Persistent workers must all be resident at once.  For CTA pairs the number of
  // co-resident clusters can be below sm_count / 2 (pairs must sit in one GPC): ask.
  static std::atomic<int> max_workers[64];
  int resident = (dev >= 0 && dev < 64) ? max_workers[dev].load(std::memory_order_acquire) : 0;
  if (resident == 0) {
    resident = sm_count() / CTAS;
    if (CTAS > 1) {
      cfg.gridDim = dim3(sm_count() / CTAS * CTAS);
      int clusters = 0;
      CK_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg));
      if (clusters > 0) resident = min(resident, clusters);
    }
    if (dev >= 0 && dev < 64) max_workers[dev].store(resident, std::memory_order_release);
  }
  int workers = min(p.tiles_m * p.tiles_n * p.splits, resident);
  if (cluster_split) workers = p.tiles_m * p.tiles_n * p.splits;  // one item per CTA
#ifdef CK_GEMM_TRACE
  if (const char* e = getenv("CK_GEMM_MAX_WORKERS")) workers = min(workers, atoi(e));
  static std::atomic<int> launch_seq{0};
  p.trace_launch = launch_seq.fetch_add(1);
#endif
  cfg.gridDim = dim3(workers * CTAS);
  CUtensorMap map_sfa = {}, map_sfb = {};
  if (CTAS == 2) {
    if (int rc = make_scale_map(&map_sfa, p.sfa, p.n_row_blocks_a, p.sf_col_tiles, Cfg::kSfTilesPerStage, 1)) return rc;
    if (int rc = make_scale_map(&map_sfb, p.sfb, p.n_row_blocks_b, p.sf_col_tiles, Cfg::kSfTilesPerStage, Cfg::kSfbRowBlocks)) return rc;
  }
  // Walking order of the tiles: the one whose concurrently running tiles touch fewer operand bytes
  // (A row blocks + B column blocks of one wave), so that a long operand is not pulled through L2
  // once per tile column (M = 16384, K = 12288: 100 MB of A per wave down the rows, 28 MB along the
  // columns).
  const int64_t a_block = static_cast<int64_t>(Cfg::kTileRows) * p.k_bytes, b_block = static_cast<int64_t>(TILE_N) * p.k_bytes;
  const int64_t w = workers, tm = p.tiles_m, tn = p.tiles_n;
  const int64_t down = (w < tm ? w : tm) * a_block + ceil_div(w, tm) * b_block;
  const int64_t along = ceil_div(w, tn) * a_block + (w < tn ? w : tn) * b_block;
  p.raster = along < down ? 1 : 0;
  OutputMaps maps_out = {};
  p.out_tma = 0;
  p.n_out = 1;
  if constexpr (OUT_STAGE != 0) {
    // TMA stores need 16-byte aligned bases and row pitch.  A single dense [M, N] result whose rows
    // start on 32-byte boundaries is written straight from registers instead (256-bit stores, whole
    // sectors): measured 1-3 % faster than staging it for TMA stores, whose shared-memory traffic
    // slows the next tile's main loop.  Multi-destination stores (all-gather, partial tiles of a split) go
    // through the staged path.
    bool ok = p.out != nullptr && (os.pitch * static_cast<int64_t>(sizeof(OutT))) % 16 == 0 &&
              (os.col_offset * static_cast<int64_t>(sizeof(OutT))) % 16 == 0;
    for (int d = 0; ok && d < os.n; ++d) ok = os.ptrs[d] != nullptr && reinterpret_cast<uintptr_t>(os.ptrs[d]) % 16 == 0;
    const bool direct = os.n == 1 && os.plain(p.N) && p.out != nullptr &&
                        (static_cast<int64_t>(p.N) * sizeof(OutT)) % 32 == 0 && reinterpret_cast<uintptr_t>(p.out) % 32 == 0;
    ok = ok && !direct && !cluster_split;  // a split-K cluster writes its result itself
    if (ok) {
      for (int d = 0; d < os.n; ++d) {
        void* base = static_cast<uint8_t*>(os.ptrs[d]) + os.col_offset * static_cast<int64_t>(sizeof(OutT));
        if (int rc = make_output_map(&maps_out.m[d], base, p.M, p.N, sizeof(OutT), os.pitch)) return rc;
      }
      p.out_tma = 1;
      p.n_out = os.n;
    }
  }
  if (p.out_tma == 0 && !os.plain(p.N)) {
    return fail(CK_ERR_INVALID_ARGUMENT, "strided or multiple outputs need 16-byte aligned buffers, pitch and column offset");
  }
  CK_CUDA(cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, map_sfa, map_sfb, maps_out, p));
  return CK_OK;
}

}  // namespace
}  // namespace ck
