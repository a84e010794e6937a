// Block-scaled GEMMs with very few activation rows (M <= 32): weight streaming.
//
// out[M, N] = x[M, K] . W[N, K]^T with M small reads the whole weight once and does almost no
// arithmetic: it is bound by HBM (0.5625 bytes per NVFP4 weight element) and by fixed latencies.
// The 128-row tile configurations spend their MMA rows, their operand loads and their epilogue on
// padding.  Here the operands change places (ck_gemm_kernel.cuh, SWAP): weight rows fill the 128
// tensor-memory lanes, the activation rows are the MMA's N (32), the accumulator is 32 columns
// wide and the epilogue writes 32 values per thread.  When the weight has few 128-row tiles and a
// long K, every tile's K range is cut over a cluster of CTAs so that all SMs stream (two CTAs fit on
// an SM); the cluster adds its partial tiles in split order through distributed shared memory.
// Measured against the tile path: wins up to 32 rows, loses from 64 rows on.
#include "ck_gemm_kernel.cuh"

namespace ck {
namespace {

constexpr int kMaxSmallM = 32;
constexpr int kSmallTileN = 32;  // the MMA's N: activation rows, padded

// CTAs per tile (1 = no split).  The most whose clusters all run at once with one CTA on an SM; with two on an SM
// when that leaves a CTA more than ten stages.  (The occupancy query counts one for every kernel that allocates
// tensor memory; two of this configuration share an SM.  A cluster that finds no room runs later: nobody waits for
// it.)  Graph replays, us, few CTAs of many stages / more: NVFP4 32 x 4096 x 12288 (12 stages / 8) 8.9 / 8.0,
// 1 x 6144 x 8192 (16 / 7) 8.9 / 8.1, 1 x 6144 x 6144 (12 / 5) 7.6 / 7.6, MXFP8 32 x 6144 x 12288 (48 / 20) 18.3 / 11.7,
// 1 x 4096 x 12288 (24 / 16) 10.9 / 9.6; but NVFP4 1 x 4096 x 8192 (8 / 6) 6.6 / 7.1, 1 x 6144 x 4096 (8 / 4) 6.2 / 6.4.
template <Kind KIND, typename OutT>
int choose_splits(int64_t N, int k_bytes, int* out) {
  const int k_stages = static_cast<int>(ceil_div(k_bytes, kStageKBytes));
  const int64_t tiles = ceil_div(N, kTileM);
  const int most = small_m_max_splits(N, k_bytes);
  constexpr int kMaxStagesAlone = 10;
  int splits = 1;
  for (int per_sm = 1; per_sm <= 2; ++per_sm) {
    for (splits = most; splits > 1; --splits) {
      int clusters = 0;
      if (int rc = split_clusters<KIND, kSmallTileN, 2, 4, OutT, 0, true>(splits, &clusters)) return rc;
      if (clusters * per_sm >= tiles) break;
    }
    if (ceil_div(k_stages, splits) <= kMaxStagesAlone) break;
  }
  *out = static_cast<int>(ceil_div(k_stages, ceil_div(k_stages, splits)));  // none without a stage
  return CK_OK;
}

template <Kind KIND, typename OutT>
int launch_small(const Operands& ops, GemmParams p, cudaStream_t stream) {
  OutputSpec os;
  void* const single[1] = {p.out};
  os.ptrs = single;
  os.n = 1;
  os.pitch = p.N;
  os.col_offset = 0;
  if (int rc = choose_splits<KIND, OutT>(p.M, p.k_bytes, &p.splits)) return rc;
  p.k_stages_per_split = static_cast<int>(ceil_div(ceil_div(p.k_bytes, kStageKBytes), p.splits));
  if (p.splits == 1) return launch_config<KIND, kSmallTileN, 2, 4, 1, OutT, false, 0, true>(ops, p, os, stream);
  // a quarter tile of one activation row per warp of the cluster, if there are warps enough for all of them
  if (4 * p.N <= p.splits * epilogue_warps(false, kSmallTileN)) {
    return launch_config<KIND, kSmallTileN, 2, 4, 1, OutT, false, 0, true, Split::kCluster>(ops, p, os, stream);
  }
  return launch_config<KIND, kSmallTileN, 2, 4, 1, OutT, false, 0, true, Split::kClusterManyRows>(ops, p, os, stream);
}

}  // namespace

bool small_m_applies(int64_t M, int64_t N, int64_t K) { return M >= 1 && M <= kMaxSmallM && N >= 1 && K >= 32; }

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

int small_m_splits(bool is_mxfp8, int out_dtype, int64_t N, int k_bytes, int* splits) {
  if (is_mxfp8) {
    switch (out_dtype) {
      case CK_DTYPE_BF16: return choose_splits<Kind::kMxfp8, __nv_bfloat16>(N, k_bytes, splits);
      case CK_DTYPE_F16: return choose_splits<Kind::kMxfp8, __half>(N, k_bytes, splits);
      default: return choose_splits<Kind::kMxfp8, float>(N, k_bytes, splits);
    }
  }
  switch (out_dtype) {
    case CK_DTYPE_BF16: return choose_splits<Kind::kNvfp4, __nv_bfloat16>(N, k_bytes, splits);
    case CK_DTYPE_F16: return choose_splits<Kind::kNvfp4, __half>(N, k_bytes, splits);
    default: return choose_splits<Kind::kNvfp4, float>(N, k_bytes, splits);
  }
}

// a: activation [M, K], b: weight [N, K] (the public argument order); shapes and pointers were validated by the caller.
int scaled_mm_small_m(bool is_mxfp8, const void* a, const void* b, const void* sfa, const void* sfb, const float* tsa,
                      const float* tsb, const float* alpha, const void* bias, int bias_dtype, void* out, int out_dtype,
                      int64_t M, int64_t N, int64_t K, cudaStream_t stream) {
  const int block = is_mxfp8 ? 32 : 16;
  GemmParams p{};
  // operands change places: the kernel's "A" is the weight
  p.sfa = static_cast<const uint8_t*>(sfb);
  p.sfb = static_cast<const uint8_t*>(sfa);
  p.tsa = tsa;
  p.tsb = tsb;
  p.alpha = alpha;
  p.bias = bias;
  p.out = out;
  p.bias_dtype = bias_dtype;
  p.out_dtype = out_dtype;
  p.M = static_cast<int>(N);
  p.N = static_cast<int>(M);
  p.k_bytes = static_cast<int>(is_mxfp8 ? K : K / 2);
  p.sf_col_tiles = static_cast<int>(ceil_div(K / block, 4));
  p.n_row_blocks_a = static_cast<int>(ceil_div(N, 128));
  p.n_row_blocks_b = static_cast<int>(ceil_div(M, 128));
  if (int rc = gemm_status_word(&p.status)) return rc;
  p.splits = 1;
  const Operands ops = {b, a};
  if (is_mxfp8) {
    switch (out_dtype) {
      case CK_DTYPE_BF16: return launch_small<Kind::kMxfp8, __nv_bfloat16>(ops, p, stream);
      case CK_DTYPE_F16: return launch_small<Kind::kMxfp8, __half>(ops, p, stream);
      default: return launch_small<Kind::kMxfp8, float>(ops, p, stream);
    }
  }
  switch (out_dtype) {
    case CK_DTYPE_BF16: return launch_small<Kind::kNvfp4, __nv_bfloat16>(ops, p, stream);
    case CK_DTYPE_F16: return launch_small<Kind::kNvfp4, __half>(ops, p, stream);
    default: return launch_small<Kind::kNvfp4, float>(ops, p, stream);
  }
}

}  // namespace ck

#ifdef CK_GEMM_TRACE
// Timeline buffers of this translation unit's kernels (see gemm_timeline.py --small-m).
extern "C" __attribute__((visibility("default"))) int ck_debug_trace_smallm(long long* host_out) {
  CK_CUDA(cudaDeviceSynchronize());
  CK_CUDA(cudaMemcpyFromSymbol(host_out, ck::g_trace, sizeof(long long) * 160 * ck::kTraceTiles * ck::kTraceSlots));
  return CK_OK;
}
extern "C" __attribute__((visibility("default"))) int ck_debug_trace3_smallm(long long* host_out) {
  CK_CUDA(cudaDeviceSynchronize());
  CK_CUDA(cudaMemcpyFromSymbol(host_out, ck::g_trace3, sizeof(long long) * 8 * 160 * 8));
  return CK_OK;
}
#endif
