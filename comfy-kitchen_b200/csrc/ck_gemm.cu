// Block-scaled GEMM entry points (scaled_mm_nvfp4 / scaled_mm_mxfp8, fused linear, split-K,
// all-gather variants): shape-based choice of the kernel configuration of
// ck_gemm_kernel.cuh, argument validation, and the device status word.
#include "ck_gemm_kernel.cuh"

namespace ck {

__device__ int g_gemm_status = 0;

// Device address of the status word on the current device (looked up once per device).
int gemm_status_word(int** out) {
  static std::atomic<int*> cached[64];
  int dev = 0;
  CK_CUDA(cudaGetDevice(&dev));
  int* ptr = (dev >= 0 && dev < 64) ? cached[dev].load(std::memory_order_acquire) : nullptr;
  if (ptr == nullptr) {
    CK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_gemm_status));
    if (dev >= 0 && dev < 64) cached[dev].store(ptr, std::memory_order_release);
  }
  *out = ptr;
  return CK_OK;
}

int forced_gemm_config() {
  // CK_GEMM_CONFIG pins the kernel configuration (used by the tests to cover each one); unset =
  // choose by shape.
  //   1 = one CTA, 128 x 128 tiles (two accumulators)   3 = one CTA, 128 x 256 tiles
  //   4 = CTA pair, 256 x 256 tiles                      7 = one CTA, 128 x 64 tiles (small problems)
  const char* e = getenv("CK_GEMM_CONFIG");
  return e ? atoi(e) : 0;
}

namespace {

// 128 x 64 tiles that find an SM each: half the columns to an epilogue, and more CTAs that load (us, 128 x 128 / 128 x 64: NVFP4 256 x 3072
// x 3072 6.5 / 6.0, 128 x 9216 x 3072 7.2 / 6.8, 1003 x 1024 x 3072 6.2 / 6.1, 384 x 3072 x 2048 5.5 / 5.4, MXFP8 128 x 9216 x 1536 7.0 / 6.6).
bool one_wave_of_half_tiles(int64_t M, int64_t N) { return ceil_div(M, kTileM) * ceil_div(N, 64) <= sm_count(); }

// Whether they pay.  Twice the CTAs ask for the same rows of the activation at once.  Rows that straddle the 128-byte lines cost each
// of them two: with one or two row blocks that is dearer (NVFP4 68 x 6304 x 2976 7.4 / 8.9, 128 x 8512 x 3808 9.8 / 10.0, 256 x 4640 x 3296 8.6 / 8.8).
// Up to 64 rows the epilogue has little to halve: from eight stages on they pay all the same (drawn sizes: 0.97 of the time up to 17 stages, 0.95
// beyond, 1.05 below eight).
bool half_tiles_pay(int64_t M, int64_t N, int k_bytes) {
  if (!one_wave_of_half_tiles(M, N)) return false;
  if (k_bytes % kStageKBytes != 0) return M > 2 * kTileM;
  return M > 64 || k_bytes >= 8 * kStageKBytes;
}

// In a linear with a dynamic scale.  Such calls in a row are a chain of reduction, quantizer and GEMM whose launches overlap, and the quantizer's
// few large blocks find room beside the GEMM before them only on SMs that it leaves free.  A GEMM of more, smaller CTAs gains less than
// the quantizer then loses, unless a quarter of the SMs stays free (whole linears, us, 128 x 128 / half tiles: 200 x 4544 x 768 7.5 / 8.6, 65 x 9216 x 3072
// 11.2 / 12.9, 1003 x 1024 x 768 8.1 / 8.7; 128 x 6848 x 3072, 107 half tiles, 11.8 / 10.7, 1003 x 576 x 352 8.6 / 7.4; pair / 128 x 128: 512 x 6848
// x 768, 54 pairs, 10.9 / 11.7, 1003 x 3072 x 512 10.8 / 11.3; 640 x 6848 x 768, 81 pairs on 74, 14.1 / 12.4).
struct Room {
  bool wanted;
  bool left_by_half_tiles(int64_t M, int64_t N) const { return !wanted || ceil_div(M, kTileM) * ceil_div(N, 64) * 4 <= 3 * sm_count(); }
};

// 128 x 128 tiles that take no more waves than pair tiles: a wave of them is shorter, with half the output of an SM behind its main loop.
// That is where the pairs' last rows or columns are padding, with 257 to 384 rows above all, or their last wave is nearly empty.  us, pair / 128 x 128:
// NVFP4 300 x 6144 x 3072 (48 pairs, 144 tiles) 9.1 / 7.1, 300 x 12288 x 3072 13.7 / 11.1, 384 x 12288 x 6144 22.3 / 18.9, MXFP8 384 x 6144 x 3072
// 13.4 / 10.5, fused 384 x 9600 x 3072 14.8 / 11.8, 1152 x 4096 x 3072 15.7 / 12.1; with one wave more 768 x 9216 x 3072 14.0 / 15.1.  In front of
// the next dynamic linear (Room) a full wave of small tiles is not worth it, 144 x 9472 x 1792 (37 pairs, 148 tiles) 12.0 / 12.9, 832 x 2560 x 3136
// (40, 140) 15.1 / 15.7, unless a sixth of the pairs' tiles is padding: 282 x 5696 x 3136 (46, 135) 15.1 / 13.6.
bool tiles_in_as_few_waves(int64_t tiles, int64_t pairs, const Room& room) {
  const int64_t tile_waves = ceil_div(tiles, sm_count()), pair_waves = ceil_div(pairs, sm_count() / 2);
  return tile_waves <= pair_waves && tile_waves <= 3 && (!room.wanted || tile_waves > 1 || 10 * pairs >= 3 * tiles);
}

// One wave more of them, while the K is so short that a tile's time is its latencies and its epilogue, which the second accumulator of a
// small tile hides.  us, pair / 128 x 128, two waves against one: NVFP4 512 x 9216 x 1280 7.9 / 7.2, x 1536 8.4 / 7.8, x 1792 8.7 / 8.6, x 2048 9.0 /
// 9.1, MXFP8 x 640 7.9 / 7.1, x 768 8.3 / 7.7, x 1024 8.9 / 8.9; three against two: 1280 x 4608 x 1280 8.9 / 8.5, x 1536 9.4 / 9.3, 700 x 9216 x 1536
// 9.5 / 9.8; four against two: 2048 x 4608 x 512 8.4 / 8.8.  The fused epilogue is the longer one: 512 x 9216 x 1536 10.8 / 10.1, x 3072 12.9 / 12.6,
// x 4096 14.4 / 14.8, 1024 x 6144 x 3072 16.4 / 16.0, 1152 x 7680 x 3072 21.8 / 19.9, but with two waves against one and up to two stages it hides
// behind nothing: 208 x 12352 x 512 8.2 / 8.7, 216 x 13440 x 256 8.1 / 8.6.  In fp32 two waves against one never pay: 384 x 9216 x 256 11.5 / 12.7,
// 640 x 4608 x 1024 12.2 / 13.1, 1024 x 4608 x 1280 13.0 / 14.0, 2048 x 2048 x 1792 13.3 / 14.5, 640 x 4608 x 3072 14.9 / 15.6; three against two pay
// as in 16 bits, 1152 x 7680 x 1280 28.8 / 24.6, 2048 x 4608 x 3072 24.3 / 24.0.  Rows of K that straddle 128-byte lines cost twice as many readers
// more (1003 x 4096 x 1248 7.7 / 8.3, MXFP8 650 x 6400 x 736 9.3 / 9.5, fused 179 x 18368 x 672 10.0 / 11.4). In front of the next dynamic linear
// only where a sixth is padding, as above: 1003 x 6144 x 1024 14.9 / 15.3, 520 x 10240 x 1024 16.4 / 14.9.
bool tiles_in_one_wave_more(int64_t tiles, int64_t pairs, int k_bytes, bool fused, bool fp32, const Room& room) {
  const int64_t tile_waves = ceil_div(tiles, sm_count()), pair_waves = ceil_div(pairs, sm_count() / 2), k_stages = ceil_div(k_bytes, kStageKBytes);
  const bool padded = 10 * pairs >= 3 * tiles;
  if (tile_waves != pair_waves + 1 || tile_waves > 4) return false;
  if (room.wanted && (tile_waves == 2 || !padded)) return false;
  if (k_bytes % kStageKBytes != 0) return !fused && tile_waves == 2 && k_stages <= 4;
  if (fused) return k_stages <= 12 && (tile_waves > 2 || (!fp32 && (k_stages >= 3 || padded)));
  return k_stages <= (tile_waves == 2 ? 6 : 5);
}

template <Kind KIND, typename OutT, bool FUSED>
int launch_for_shape(const Operands& ops, const GemmParams& p, const OutputSpec& os, const Room& room, cudaStream_t stream) {
  int config = forced_gemm_config();
  if (config == 0) {
    const int64_t row_blocks = ceil_div(p.M, kTileM), tiles = row_blocks * ceil_div(p.N, 128);
    // The pair, from about a quarter of the SM count in pair tiles on: not where its second CTA would have no rows (us, pair / 128 x 128,
    // NVFP4 128 x 18432 x 1024 8.0 / 6.0, x 3072 11.4 / 9.4, x 8192 20.1 / 18.3, 128 x 36864 x 3072 17.1 / 15.1, MXFP8 128 x 18432 x 3072
    // 16.5 / 13.8, the fused epilogue 128 x 12288 x 3072 12.6 / 9.1), and not where small tiles beat it (above).
    const int64_t pairs = ceil_div(p.M, 256) * ceil_div(p.N, 256);
    const bool pair = pairs * 4 >= sm_count() && row_blocks > 1 && !tiles_in_as_few_waves(tiles, pairs, room) &&
                      !tiles_in_one_wave_more(tiles, pairs, p.k_bytes, FUSED, sizeof(OutT) == 4, room);
    if (pair) {
      config = 4;
    } else if (tiles * 4 <= sm_count() || (half_tiles_pay(p.M, p.N, p.k_bytes) && room.left_by_half_tiles(p.M, p.N))) {
      config = 7;
    } else {
      config = 1;
    }
  }
  // strided / multiple destinations exist only in the configurations with a staged epilogue
  if (!os.plain(p.N) && config != 4 && config != 7) config = 1;
  switch (config) {
    case 7:
      if constexpr (!FUSED) return launch_config<KIND, 64, 2, 6, 1, OutT, false, 1>(ops, p, os, stream);
      return launch_config<KIND, 128, 2, 6, 1, OutT, FUSED>(ops, p, os, stream);
    case 4:
      return launch_config<KIND, 256, 1, 5, 2, OutT, FUSED, FUSED ? 0 : 1>(ops, p, os, stream);
    case 3:
      return launch_config<KIND, 256, 1, 4, 1, OutT, FUSED>(ops, p, os, stream);
    default:
      if constexpr (!FUSED) return launch_config<KIND, 128, 2, 5, 1, OutT, false, 1>(ops, p, os, stream);
      return launch_config<KIND, 128, 2, 6, 1, OutT, FUSED>(ops, p, os, stream);
  }
}

// ---------------------------------------------------------------------------
// split-K
// ---------------------------------------------------------------------------
// Few 128 x 128 tiles and a long K: the K range of a tile is spread over several CTAs.  At most as many as fit the
// chip and leave every CTA six pipeline stages; 1 = no split, also where only two CTAs would come of it (below 18
// stages; graph replays, us, split in two / unsplit: NVFP4 128 x 3072 x 4096 8.3 / 7.3, 256 x 4096 x 4096 8.7 / 7.9).
int max_splits(int64_t M, int64_t N, int k_bytes) {
  const int k_stages = static_cast<int>(ceil_div(k_bytes, kStageKBytes));
  const int64_t tiles = ceil_div(M, kTileM) * ceil_div(N, 128);
  if (tiles * 2 > sm_count() || k_stages < 18) return 1;
  int splits = min(kMaxSplits, k_stages / 6);
  const int64_t by_sms = sm_count() / tiles;
  if (by_sms < splits) splits = static_cast<int>(by_sms);
  return max(splits, 1);
}

struct SplitPlan {
  int splits;            // CTAs per tile; 1:
  bool half_tiles;       //   tiles of half the columns instead of two CTAs to one
  int k_stages;          // of each
  bool through_workspace;
};

int64_t split_workspace_bytes(int64_t M, int64_t N, const SplitPlan& plan) { return plan.splits * M * N * 4; }

// A cluster of CTAs adds its partial tiles on chip (ck_gemm_kernel.cuh): the most CTAs per tile whose clusters all run
// at once.  A cluster sits in one part of the chip, which can leave SMs idle that a split without clusters uses; its
// CTAs store their partial tiles to a workspace and a second kernel adds them.  That exchange costs about four
// thirds of a pipeline stage per partial tile, so it is taken where it saves a CTA that many.  Graph replays, us,
// clusters / workspace: 256 x 3072 x 12288 13.3 / 12.8 with NVFP4 (24 / 16 stages, 3 partial tiles), 19.5 / 16.7 with MXFP8
// (48 / 32), x 6144 NVFP4 9.8 / 10.0 (12 / 8), 256 x 2176 x 12288 MXFP8 14.8 / 14.2 (32 / 24, 4); but 256 x 2176 x 12288 NVFP4
// 10.7 / 11.3 (16 / 12, 4), 256 x 1152 x 12288 MXFP8 10.9 / 11.7 (16 / 12, 8), 128 x 3712 x 16384 MXFP8 17.5 / 18.1 (32 / 26, 5).
template <Kind KIND, typename OutT>
int choose_splits(int64_t M, int64_t N, int k_bytes, bool have_workspace, SplitPlan* plan) {
  const int64_t tiles = ceil_div(M, kTileM) * ceil_div(N, 128);
  const int k_stages = static_cast<int>(ceil_div(k_bytes, kStageKBytes));
  const int most = max_splits(M, N, k_bytes);
  int splits = most;
  for (; splits > 1; --splits) {
    int clusters = 0;
    if (int rc = split_clusters<KIND, 128, 2, 5, OutT, 1>(splits, &clusters)) return rc;
    if (clusters >= tiles) break;
  }
  plan->through_workspace = have_workspace && 3 * (ceil_div(k_stages, splits) - ceil_div(k_stages, most)) >= 4 * most && most > 1;
  // Two CTAs to a tile: half tiles instead, while their longer K costs less than the exchange.  They end in TMA stores, which want
  // rows of whole 64-byte units (N of 16 bits off by 16: MXFP8 512 x 1648 x 2784 10.0 / 10.7, NVFP4 517 x 1584 x 4800 9.7 / 10.7).  us, two CTAs /
  // half tiles: linears NVFP4 256 x 4608, 24 stages, 12.9 / 11.5, 300 x 2048, 24 stages, 12.3 / 11.4, MXFP8 256 x 4608, 30 stages, 12.9 / 12.0.  Over
  // drawn sizes of both formats half tiles take 0.91 to 1.0 of the time from 24 to 35 stages, 1.0 from 36 to 41 and 1.05 from 42 on. Up to 64 rows
  // not where those of K straddle 128-byte lines (NVFP4 40 x 8192 x 6112 10.2 / 10.8; 64 x 8192 x 6144 10.1 / 9.4, MXFP8 64 x 9216 x 3072 10.3 /
  // 9.3).
  constexpr int kMostStages = 36;
  plan->half_tiles = splits == 2 && !plan->through_workspace && k_stages <= kMostStages && N % 32 == 0 && (M > 64 || k_bytes % kStageKBytes == 0) && one_wave_of_half_tiles(M, N);
  if (plan->half_tiles) splits = 1;
  plan->k_stages = static_cast<int>(ceil_div(k_stages, plan->through_workspace ? most : splits));
  plan->splits = static_cast<int>(ceil_div(k_stages, plan->k_stages));  // none without a stage
  return CK_OK;
}

// out = cast(alpha * (partial_0 + partial_1 + ...) + bias), four consecutive columns per thread; the partials are
// added in index order, so the result does not depend on scheduling.
template <typename OutT>
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* partials, int splits, int64_t mn, int n_cols, const float* alpha_ptr, const float* tsa,
                     const float* tsb, const void* bias, int bias_dtype, OutT* out) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (i >= mn) return;
  float alpha = 1.0f;
  if (alpha_ptr != nullptr) {
    alpha = ld_f32_dependent(alpha_ptr);
  } else if (tsa != nullptr && tsb != nullptr) {
    alpha = ld_f32_dependent(tsa) * ld_f32_dependent(tsb);
  }
  float4 acc = *reinterpret_cast<const float4*>(partials + i);
  for (int s = 1; s < splits; ++s) {
    const float4 v = *reinterpret_cast<const float4*>(partials + s * mn + i);
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  }
  const int n = static_cast<int>(i % n_cols);  // N % 8 == 0: a group of four never straddles two rows
  float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = load_bias(bias, bias_dtype, n + j);
  }
  const float y[4] = {fmaf(acc.x, alpha, b[0]), fmaf(acc.y, alpha, b[1]), fmaf(acc.z, alpha, b[2]), fmaf(acc.w, alpha, b[3])};
  store_four(out + i, y);
}

template <Kind KIND, typename OutT>
int launch_split(const Operands& ops, GemmParams p, const OutputSpec& os, void* workspace, int64_t workspace_bytes, bool* launched,
                 cudaStream_t stream) {
  *launched = false;
  SplitPlan plan = {};
  if (int rc = choose_splits<KIND, OutT>(p.M, p.N, p.k_bytes, workspace != nullptr, &plan)) return rc;
  if (plan.through_workspace && (workspace_bytes < split_workspace_bytes(p.M, p.N, plan) || reinterpret_cast<uintptr_t>(workspace) % 16 != 0)) {
    if (int rc = choose_splits<KIND, OutT>(p.M, p.N, p.k_bytes, false, &plan)) return rc;
  }
  *launched = plan.splits > 1 || plan.half_tiles;
  if (plan.half_tiles) return launch_config<KIND, 64, 2, 6, 1, OutT, false, 1>(ops, p, os, stream);
  if (plan.splits < 2) return CK_OK;
  const int64_t mn = static_cast<int64_t>(p.M) * p.N;
  const GemmParams result = p;
  p.splits = plan.splits;
  p.k_stages_per_split = plan.k_stages;
  if (!plan.through_workspace) return launch_config<KIND, 128, 2, 5, 1, OutT, false, 1, Split::kCluster>(ops, p, os, stream);
  p.tsa = p.tsb = p.alpha = nullptr;
  p.bias = nullptr;
  p.out = workspace;
  p.out_dtype = CK_DTYPE_F32;
  void* parts[kMaxOutputs] = {};
  for (int i = 0; i < plan.splits; ++i) parts[i] = static_cast<float*>(workspace) + i * mn;
  OutputSpec partials;
  partials.ptrs = parts;
  partials.n = plan.splits;
  partials.pitch = p.N;
  partials.col_offset = 0;
  if (int rc = launch_config<KIND, 128, 2, 5, 1, float, false, 1, Split::kOutputs>(ops, p, partials, stream)) return rc;
  CK_CUDA(launch_pdl(splitk_reduce_kernel<OutT>, dim3(static_cast<unsigned>(ceil_div(mn / 4, 256))), dim3(256), 0, stream,
                     static_cast<const float*>(workspace), plan.splits, mn, p.N, result.alpha, result.tsa, result.tsb, result.bias,
                     result.bias_dtype, static_cast<OutT*>(result.out)));
  return CK_OK;
}

template <Kind KIND>
int tile_plan(int out_dtype, int64_t M, int64_t N, int k_bytes, bool have_workspace, SplitPlan* plan) {
  switch (out_dtype) {
    case CK_DTYPE_BF16: return choose_splits<KIND, __nv_bfloat16>(M, N, k_bytes, have_workspace, plan);
    case CK_DTYPE_F16: return choose_splits<KIND, __half>(M, N, k_bytes, have_workspace, plan);
    default: return choose_splits<KIND, float>(M, N, k_bytes, have_workspace, plan);
  }
}

int tile_plan(bool is_mxfp8, int out_dtype, int64_t M, int64_t N, int64_t K, bool have_workspace, SplitPlan* plan) {
  const int k_bytes = static_cast<int>(is_mxfp8 ? K : K / 2);
  return is_mxfp8 ? tile_plan<Kind::kMxfp8>(out_dtype, M, N, k_bytes, have_workspace, plan)
                  : tile_plan<Kind::kNvfp4>(out_dtype, M, N, k_bytes, have_workspace, plan);
}

struct FusedArgs {
  bool enabled = false;
  int activation = CK_ACT_NONE;
  void* rq_codes = nullptr;
  void* rq_scales = nullptr;
  const float* rq_scale = nullptr;
};

template <Kind KIND>
int scaled_mm(const char* op, const void* a, const void* b, const void* sfa, const void* sfb, const float* tsa,
              const float* tsb, const float* alpha, const void* bias, int bias_dtype, void* out, int out_dtype,
              int64_t M, int64_t N, int64_t K, void* stream, const FusedArgs& fused = FusedArgs(),
              const OutputSpec* out_spec = nullptr, void* workspace = nullptr, int64_t workspace_bytes = 0, const Room& room = Room{false}) {
  CK_REQUIRE(a && b && sfa && sfb, "%s: null pointer", op);
  CK_REQUIRE(out != nullptr || (fused.enabled && fused.rq_codes != nullptr), "%s: no output requested", op);
  if (fused.enabled) {
    CK_REQUIRE(fused.activation == CK_ACT_NONE || fused.activation == CK_ACT_GELU_TANH, "%s: unknown activation %d", op,
               fused.activation);
    if (fused.rq_codes != nullptr) {
      CK_REQUIRE(fused.rq_scales != nullptr && fused.rq_scale != nullptr, "%s: re-quantization needs scales", op);
      CK_REQUIRE(N % 64 == 0, "%s: re-quantized output needs N %% 64 == 0, got %lld", op, (long long)N);
      CK_REQUIRE(reinterpret_cast<uintptr_t>(fused.rq_codes) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(fused.rq_scales) % 4 == 0,
                 "%s: re-quantized outputs must be 16-byte (codes) and 4-byte (scales) aligned", op);
    }
  }
  CK_REQUIRE(M > 0 && N > 0 && K > 0, "%s: empty problem M=%lld N=%lld K=%lld", op, (long long)M, (long long)N,
             (long long)K);
  CK_REQUIRE(M < (1ll << 30) && N < (1ll << 30) && K < (1ll << 30), "%s: dimension too large", op);
  CK_REQUIRE(K % 32 == 0, "%s: K=%lld must be a multiple of 32", op, (long long)K);
  CK_REQUIRE(N % 8 == 0, "%s: N=%lld must be a multiple of 8", op, (long long)N);
  CK_REQUIRE(out_dtype == CK_DTYPE_F32 || out_dtype == CK_DTYPE_F16 || out_dtype == CK_DTYPE_BF16,
             "%s: unsupported output dtype code %d", op, out_dtype);
  CK_REQUIRE(bias == nullptr || bias_dtype == CK_DTYPE_F32 || bias_dtype == CK_DTYPE_F16 || bias_dtype == CK_DTYPE_BF16,
             "%s: unsupported bias dtype code %d", op, bias_dtype);
  CK_REQUIRE(reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(b) % 16 == 0,
             "%s: operands must be 16-byte aligned", op);
  CK_REQUIRE(reinterpret_cast<uintptr_t>(sfa) % 16 == 0 && reinterpret_cast<uintptr_t>(sfb) % 16 == 0,
             "%s: block scales must be 16-byte aligned", op);
  if (KIND == Kind::kNvfp4) CK_REQUIRE(alpha != nullptr || (tsa != nullptr && tsb != nullptr), "%s: null tensor scale", op);

  const int block = (KIND == Kind::kNvfp4) ? 16 : 32;
  GemmParams p{};
  p.sfa = static_cast<const uint8_t*>(sfa);
  p.sfb = static_cast<const uint8_t*>(sfb);
  p.tsa = tsa;
  p.tsb = tsb;
  p.alpha = alpha;
  p.bias = bias;
  p.out = out;
  p.bias_dtype = bias_dtype;
  p.out_dtype = out_dtype;
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.k_bytes = static_cast<int>(KIND == Kind::kNvfp4 ? K / 2 : K);
  p.sf_col_tiles = static_cast<int>(ceil_div(K / block, 4));
  p.activation = fused.activation;
  p.rq_codes = static_cast<uint8_t*>(fused.rq_codes);
  p.rq_scales = static_cast<uint8_t*>(fused.rq_scales);
  p.rq_scale = fused.rq_scale;
  p.n_row_blocks_a = static_cast<int>(ceil_div(M, 128));
  p.n_row_blocks_b = static_cast<int>(ceil_div(N, 128));
  p.splits = 1;
  p.k_stages_per_split = static_cast<int>(ceil_div(p.k_bytes, kStageKBytes));
  if (int rc = gemm_status_word(&p.status)) return rc;
  const Operands ops = {a, b};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  OutputSpec os;
  void* const single[1] = {out};
  if (out_spec != nullptr) {
    os = *out_spec;
    CK_REQUIRE(!fused.enabled, "%s: the fused epilogue has one plain output", op);
    CK_REQUIRE(os.n >= 1 && os.n <= kMaxOutputs && os.ptrs != nullptr, "%s: 1..%d output buffers", op, kMaxOutputs);
    CK_REQUIRE(os.col_offset >= 0 && os.col_offset + N <= os.pitch, "%s: columns [%lld, %lld) outside a pitch of %lld", op,
               (long long)os.col_offset, (long long)(os.col_offset + N), (long long)os.pitch);
  } else {
    os.ptrs = single;
    os.n = 1;
    os.pitch = N;
    os.col_offset = 0;
  }
  if (!fused.enabled && out_spec == nullptr) {
    // Few activation rows: the weight-streaming path (weight rows in the MMA's M, K split over clusters).
    // CK_GEMM_CONFIG=9 forces it, any other forced configuration keeps it off.
    if (small_m_applies(M, N, K) && (forced_gemm_config() == 0 || forced_gemm_config() == 9)) {
      return scaled_mm_small_m(KIND == Kind::kMxfp8, a, b, sfa, sfb, tsa, tsb, alpha, bias, bias_dtype, out, out_dtype, M, N, K, s);
    }
    // the rows of the result are written four columns at a time
    if (max_splits(M, N, p.k_bytes) > 1 && forced_gemm_config() == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0) {
      bool launched = false;
      int rc = CK_OK;
      switch (out_dtype) {
        case CK_DTYPE_BF16: rc = launch_split<KIND, __nv_bfloat16>(ops, p, os, workspace, workspace_bytes, &launched, s); break;
        case CK_DTYPE_F16: rc = launch_split<KIND, __half>(ops, p, os, workspace, workspace_bytes, &launched, s); break;
        default: rc = launch_split<KIND, float>(ops, p, os, workspace, workspace_bytes, &launched, s);
      }
      if (rc != CK_OK || launched) return rc;
    }
  }
  if constexpr (KIND == Kind::kNvfp4) {
    if (fused.enabled) {
      switch (out_dtype) {
        case CK_DTYPE_BF16:
          return launch_for_shape<KIND, __nv_bfloat16, true>(ops, p, os, room, s);
        case CK_DTYPE_F16:
          return launch_for_shape<KIND, __half, true>(ops, p, os, room, s);
        default:
          return launch_for_shape<KIND, float, true>(ops, p, os, room, s);
      }
    }
  }
  switch (out_dtype) {
    case CK_DTYPE_BF16:
      return launch_for_shape<KIND, __nv_bfloat16, false>(ops, p, os, room, s);
    case CK_DTYPE_F16:
      return launch_for_shape<KIND, __half, false>(ops, p, os, room, s);
    default:
      return launch_for_shape<KIND, float, false>(ops, p, os, room, s);
  }
}

}  // namespace

int scaled_mm_of_dynamic_linear(const void* a, const void* b, const void* sfa, const void* sfb, const float* tsa, const float* tsb, const void* bias,
                                int bias_dtype, void* out, int out_dtype, int64_t M, int64_t N, int64_t K, void* stream) {
  return scaled_mm<Kind::kNvfp4>("scaled_mm_nvfp4", a, b, sfa, sfb, tsa, tsb, nullptr, bias, bias_dtype, out, out_dtype, M, N, K, stream, FusedArgs(),
                                 nullptr, nullptr, 0, Room{true});
}

}  // namespace ck

extern "C" int ck_scaled_mm_nvfp4(const void* a, const void* b, const void* sfa, const void* sfb,
                                  const float* tensor_scale_a, const float* tensor_scale_b, const float* alpha,
                                  const void* bias, int bias_dtype, void* out, int out_dtype, int64_t M, int64_t N,
                                  int64_t K, void* stream) {
  return ck::scaled_mm<ck::Kind::kNvfp4>("scaled_mm_nvfp4", a, b, sfa, sfb, tensor_scale_a, tensor_scale_b, alpha, bias,
                                         bias_dtype, out, out_dtype, M, N, K, stream);
}

extern "C" int ck_scaled_mm_mxfp8(const void* a, const void* b, const void* sfa, const void* sfb, const void* bias,
                                  int bias_dtype, void* out, int out_dtype, int64_t M, int64_t N, int64_t K,
                                  void* stream) {
  return ck::scaled_mm<ck::Kind::kMxfp8>("scaled_mm_mxfp8", a, b, sfa, sfb, nullptr, nullptr, nullptr, bias, bias_dtype,
                                         out, out_dtype, M, N, K, stream);
}

extern "C" int ck_linear_nvfp4_fused(const void* a, const void* b, const void* sfa, const void* sfb,
                                     const float* tensor_scale_a, const float* tensor_scale_b, const float* alpha,
                                     const void* bias, int bias_dtype, int activation, void* out, int out_dtype,
                                     void* requant_codes, void* requant_block_scales, const float* requant_scale,
                                     int64_t M, int64_t N, int64_t K, void* stream) {
  ck::FusedArgs f;
  f.enabled = true;
  f.activation = activation;
  f.rq_codes = requant_codes;
  f.rq_scales = requant_block_scales;
  f.rq_scale = requant_scale;
  return ck::scaled_mm<ck::Kind::kNvfp4>("linear_nvfp4_fused", a, b, sfa, sfb, tensor_scale_a, tensor_scale_b, alpha, bias,
                                         bias_dtype, out, out_dtype, M, N, K, stream, f);
}

// Non-zero for the shapes whose K may be split: kOnChip where the partial tiles stay on chip (or K is long, but not
// long enough), which callers of this query have been given for those shapes before and which is not used.
extern "C" int64_t ck_scaled_mm_workspace_bytes(int is_mxfp8, int64_t M, int64_t N, int64_t K) {
  using namespace ck;
  constexpr int64_t kOnChip = 256;
  if (M <= 0 || N <= 0 || K <= 0 || M >= (1ll << 30) || N >= (1ll << 30) || K >= (1ll << 30)) return 0;
  const int k_bytes = static_cast<int>(is_mxfp8 ? K : K / 2);
  if (small_m_applies(M, N, K)) return small_m_max_splits(N, k_bytes) > 1 ? kOnChip : 0;
  if (ceil_div(M, kTileM) * ceil_div(N, 128) * 2 > sm_count() || ceil_div(k_bytes, kStageKBytes) < 16) return 0;
  SplitPlan plan = {};
  if (tile_plan(is_mxfp8 != 0, CK_DTYPE_BF16, M, N, K, true, &plan) != CK_OK || !plan.through_workspace) return kOnChip;
  return split_workspace_bytes(M, N, plan);
}

extern "C" int ck_debug_gemm_splits(int is_mxfp8, int out_dtype, int64_t M, int64_t N, int64_t K, int with_workspace) {
  using namespace ck;
  if (M <= 0 || N <= 0 || K <= 0 || M >= (1ll << 30) || N >= (1ll << 30) || K >= (1ll << 30)) {
    return -fail(CK_ERR_INVALID_ARGUMENT, "debug_gemm_splits: bad shape");
  }
  SplitPlan plan = {};
  const int rc = small_m_applies(M, N, K)
                     ? small_m_splits(is_mxfp8 != 0, N, static_cast<int>(is_mxfp8 ? K : K / 2), &plan.splits)
                     : tile_plan(is_mxfp8 != 0, out_dtype, M, N, K, with_workspace != 0, &plan);
  return rc == CK_OK ? plan.splits : -rc;
}

extern "C" int ck_scaled_mm_nvfp4_ws(const void* a, const void* b, const void* sfa, const void* sfb,
                                     const float* tensor_scale_a, const float* tensor_scale_b, const float* alpha,
                                     const void* bias, int bias_dtype, void* out, int out_dtype, int64_t M, int64_t N,
                                     int64_t K, void* workspace, int64_t workspace_bytes, void* stream) {
  return ck::scaled_mm<ck::Kind::kNvfp4>("scaled_mm_nvfp4", a, b, sfa, sfb, tensor_scale_a, tensor_scale_b, alpha, bias,
                                         bias_dtype, out, out_dtype, M, N, K, stream, ck::FusedArgs(), nullptr, workspace,
                                         workspace_bytes);
}

extern "C" int ck_scaled_mm_mxfp8_ws(const void* a, const void* b, const void* sfa, const void* sfb, const void* bias,
                                     int bias_dtype, void* out, int out_dtype, int64_t M, int64_t N, int64_t K,
                                     void* workspace, int64_t workspace_bytes, void* stream) {
  return ck::scaled_mm<ck::Kind::kMxfp8>("scaled_mm_mxfp8", a, b, sfa, sfb, nullptr, nullptr, nullptr, bias, bias_dtype,
                                         out, out_dtype, M, N, K, stream, ck::FusedArgs(), nullptr, workspace,
                                         workspace_bytes);
}

extern "C" int ck_scaled_mm_nvfp4_allgather(const void* a, const void* b, const void* sfa, const void* sfb,
                                            const float* tensor_scale_a, const float* tensor_scale_b, const float* alpha,
                                            const void* bias, int bias_dtype, void* const* out_ptrs, int world,
                                            int out_dtype, int64_t M, int64_t N_local, int64_t K, int64_t n_total,
                                            int64_t col_offset, void* stream) {
  ck::OutputSpec os;
  os.ptrs = out_ptrs;
  os.n = world;
  os.pitch = n_total;
  os.col_offset = col_offset;
  CK_REQUIRE(out_ptrs != nullptr && world >= 1 && world <= ck::kMaxOutputs, "scaled_mm_nvfp4_allgather: 1..%d destinations",
             ck::kMaxOutputs);
  return ck::scaled_mm<ck::Kind::kNvfp4>("scaled_mm_nvfp4_allgather", a, b, sfa, sfb, tensor_scale_a, tensor_scale_b, alpha,
                                         bias, bias_dtype, out_ptrs[0], out_dtype, M, N_local, K, stream, ck::FusedArgs(), &os);
}

extern "C" int ck_scaled_mm_mxfp8_allgather(const void* a, const void* b, const void* sfa, const void* sfb,
                                            const void* bias, int bias_dtype, void* const* out_ptrs, int world,
                                            int out_dtype, int64_t M, int64_t N_local, int64_t K, int64_t n_total,
                                            int64_t col_offset, void* stream) {
  ck::OutputSpec os;
  os.ptrs = out_ptrs;
  os.n = world;
  os.pitch = n_total;
  os.col_offset = col_offset;
  CK_REQUIRE(out_ptrs != nullptr && world >= 1 && world <= ck::kMaxOutputs, "scaled_mm_mxfp8_allgather: 1..%d destinations",
             ck::kMaxOutputs);
  return ck::scaled_mm<ck::Kind::kMxfp8>("scaled_mm_mxfp8_allgather", a, b, sfa, sfb, nullptr, nullptr, nullptr, bias,
                                         bias_dtype, out_ptrs[0], out_dtype, M, N_local, K, stream, ck::FusedArgs(), &os);
}

#ifdef CK_GEMM_TRACE
// Copies the per-tile timeline to the host: [160 CTAs][40 tiles][16 slots] of SM cycle counts.
extern "C" __attribute__((visibility("default"))) int ck_debug_trace(long long* host_out) {
  CK_CUDA(cudaDeviceSynchronize());
  CK_CUDA(cudaMemcpyFromSymbol(host_out, ck::g_trace, sizeof(long long) * 160 * ck::kTraceTiles * ck::kTraceSlots));
  return CK_OK;
}
extern "C" __attribute__((visibility("default"))) int ck_debug_trace3(long long* host_out) {
  CK_CUDA(cudaDeviceSynchronize());
  CK_CUDA(cudaMemcpyFromSymbol(host_out, ck::g_trace3, sizeof(long long) * 8 * 160 * 8));
  return CK_OK;
}
extern "C" __attribute__((visibility("default"))) int ck_debug_trace2(long long* host_out) {
  CK_CUDA(cudaDeviceSynchronize());
  CK_CUDA(cudaMemcpyFromSymbol(host_out, ck::g_trace2, sizeof(long long) * 160 * 4 * 64));
  return CK_OK;
}
#endif

// Validation aid: sets the status word from the host, so that the error path of callers can be
// tested without making a kernel fail.
extern "C" int ck_debug_set_gemm_status(int value) {
  CK_CUDA(cudaDeviceSynchronize());
  CK_CUDA(cudaMemcpyToSymbol(ck::g_gemm_status, &value, sizeof(int)));
  return CK_OK;
}

// Device status word of the GEMM kernels: 0 = every wait completed; non-zero = some wait
// gave up (results of that launch are invalid).  Synchronises the device; resets the word.
extern "C" int ck_gemm_status(int* status_out) {
  int v = 0;
  CK_CUDA(cudaDeviceSynchronize());
  CK_CUDA(cudaMemcpyFromSymbol(&v, ck::g_gemm_status, sizeof(int)));
  if (v != 0) {
    const int zero = 0;
    CK_CUDA(cudaMemcpyToSymbol(ck::g_gemm_status, &zero, sizeof(int)));
  }
  if (status_out != nullptr) *status_out = v;
  return CK_OK;
}
