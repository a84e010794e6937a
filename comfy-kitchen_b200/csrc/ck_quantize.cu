// Block quantizers for sm_100a: bf16/f16/f32 -> NVFP4 (E2M1 codes + E4M3 scales per
// 16 elements) and -> MXFP8 (E4M3 data + E8M0 scales per 32 elements), both with the
// scale bytes written straight into the 128x4-tiled layout the tensor cores consume.
//
// Both kernels are streaming kernels whose floor is HBM bandwidth.  One thread owns one scale
// block of one row (2-D block and grid indices, no integer division), so a warp reads 32
// consecutive blocks (1 KiB / 2 KiB of bf16) with 256-bit loads,
// writes 256 B / 1 KiB of codes with 64-bit / 256-bit stores, and the four lanes that
// share a 4-byte group of the scale tile merge their bytes by shuffle into one 32-bit
// store.  The thread grid spans the *padded* scale tensor so that its padding bytes are
// written as zero by the same launch (no separate memset).
//
// Arithmetic contract: results are bit-identical to the reference's eager path
// (comfy_kitchen/backends/eager/quantization.py:115-160 and :257-324), which uses true
// IEEE fp32 divisions.  This translation unit is therefore compiled without fast-math,
// and every division below is __fdiv_rn, a reciprocal-FMA sequence that is proven to round
// identically (see div_markstein), or none at all where what it is rounded to is certain without
// it: an E2M1 code by a corrected quotient (16-bit inputs, nvfp4_codes_corrected), a code or an E4M3
// scale by two products on either side of the quotient (nvfp4_blocks).
#include "ck_quant_math.cuh"

#include <atomic>
#include <cstdlib>
#include <type_traits>

namespace ck {
namespace {

using namespace quant;

constexpr int kColsPerBlock = 64;  // scale columns per thread block (two warps wide)
constexpr int kRowsPerBlock = 4;
constexpr int kThreads = kColsPerBlock * kRowsPerBlock;

// ---------------------------------------------------------------------------
// loading N consecutive elements of one row as exact float values
// ---------------------------------------------------------------------------
template <typename T>
struct SrcTraits;
template <>
struct SrcTraits<__nv_bfloat16> {
  __device__ static float to_f32(const __nv_bfloat16& v) { return __bfloat162float(v); }
};
template <>
struct SrcTraits<__half> {
  __device__ static float to_f32(const __half& v) { return __half2float(v); }
};
template <>
struct SrcTraits<float> {
  __device__ static float to_f32(const float& v) { return v; }
};

// 16 consecutive elements starting at `p` (32-byte aligned for 2-byte types).
template <typename T>
__device__ __forceinline__ void load16_vec(const T* p, float (&v)[16]) {
  if constexpr (sizeof(T) == 2) {
    const Vec256 raw = ld_global_stream_256(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        v[2 * i] = __uint_as_float(raw.w[i] << 16);
        v[2 * i + 1] = __uint_as_float(raw.w[i] & 0xFFFF0000u);
      } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&raw.w[i]));
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
      }
    }
  } else {
    const Vec256 lo = ld_global_stream_256(p);
    const Vec256 hi = ld_global_stream_256(p + 8);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = __uint_as_float(lo.w[i]);
      v[8 + i] = __uint_as_float(hi.w[i]);
    }
  }
}

// Same, element by element with bounds checks (ragged or misaligned inputs).
template <typename T>
__device__ __forceinline__ void load16_guarded(const T* base, int64_t row, int64_t col0, int64_t rows, int64_t cols,
                                               float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int64_t c = col0 + i;
    v[i] = (row < rows && c < cols) ? SrcTraits<T>::to_f32(base[row * cols + c]) : 0.0f;
  }
}

// Executed by every lane of the warp; lanes past the padded width (`inside` false) do not store.
__device__ __forceinline__ void store_scale_quad(uint8_t* scales, int64_t row, int64_t sc, int64_t col_tiles,
                                                 uint32_t byte, bool inside) {
  uint32_t w = byte | (__shfl_xor_sync(0xFFFFFFFFu, byte, 1) << 8);
  w |= __shfl_xor_sync(0xFFFFFFFFu, w, 2) << 16;
  if (inside && (sc & 3) == 0) {
    *reinterpret_cast<uint32_t*>(scales + swizzled_scale_offset(row, sc, col_tiles)) = w;
  }
}

// A thread owns one (row, scale column) of the padded scale tensor [rows_pad, sc_pad]:
// block = (kColsPerBlock scale columns, kRowsPerBlock rows), grid = (row groups, column
// chunks).  sc_pad is a multiple of 4 and a warp is 32 consecutive scale columns of one
// row, so aligned lane quads share a row and a 4-byte scale group.
template <typename T, bool kVec, bool kFastDiv>
__global__ void __launch_bounds__(kThreads)
quantize_nvfp4_kernel(const T* x, const float* global_scale, uint8_t* __restrict__ codes,
                      uint8_t* __restrict__ scales, int64_t orig_rows, int64_t orig_cols, int64_t num_rows,
                      int64_t num_cols, int64_t sc_pad, int hi_first) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t sc = blockIdx.y * kColsPerBlock + threadIdx.x;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kRowsPerBlock + threadIdx.y;
  const int64_t n_sc = num_cols >> 4;
  uint32_t scale_byte = 0;
  if (row < num_rows && sc < n_sc) {
    float v[16];
    if constexpr (kVec) {
      load16_vec(x + row * orig_cols + sc * 16, v);
    } else {
      load16_guarded(x, row, sc * 16, orig_rows, orig_cols, v);
    }
    const float g = ld_f32_dependent(global_scale);
    uint32_t lo, hi;
    nvfp4_block<kFastDiv>(v, g, hi_first != 0, lo, hi, scale_byte);
    *reinterpret_cast<uint2*>(codes + row * (num_cols >> 1) + sc * 8) = make_uint2(lo, hi);
  }
  store_scale_quad(scales, row, sc, sc_pad >> 2, scale_byte, sc < sc_pad);
}

// Where a launch of the streaming quantizer takes its per-tensor scale from.
struct ScaleSource {
  const float* given;      // static scale, or null: amax(|x|) / 2688 of this very input, from
  const float* partials;   //   the maxima a reduction pass left (ck_amax.cu), or, when there are none,
  int n_partials;          //   the whole (small) input, which every block then reads for itself
  int64_t n_vecs;          // 32-byte units of the input
  float* out;              // the dynamic scale for whoever needs it next
  bool backward;           // begin with the last rows (walk_of)
};

// amax(|x|) / (448 * 6) of the whole input, by every block for itself (all threads return it).  NaNs
// are dropped the way nvfp4_tensor_scale_kernel drops them: both reduce the same 32-byte units.
template <typename T>
__device__ __forceinline__ float block_dynamic_scale(const T* x, const ScaleSource& src, int tid, int threads) {
  float m = 0.0f;
  if (src.n_partials > 0) {
    for (int i = tid; i < src.n_partials; i += 8 * threads) {  // eight loads in flight: there may be thousands
      float p[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) p[j] = i + j * threads < src.n_partials ? ld_f32_dependent(src.partials + i + j * threads) : 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, p[j]);
    }
  } else {
    constexpr int kPerVec = 32 / sizeof(T);
    for (int64_t i = tid; i < src.n_vecs; i += 4 * threads) {
      Vec256 raw[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        raw[j] = i + j * threads < src.n_vecs ? ld_global_stream_256(x + (i + j * threads) * kPerVec) : Vec256{};
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) m = fmaxf(m, abs_max_of_vec<T>(raw[j]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  __shared__ float warp_max[32];
  if ((tid & 31) == 0) warp_max[tid >> 5] = m;
  __syncthreads();
  m = (tid & 31) < threads / 32 ? warp_max[tid & 31] : 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  return nvfp4_scale_of_amax<T>(m);
}

// Streaming kernel for inputs whose rows are whole 64-byte units (two scale blocks of a 16-bit type,
// one of fp32) and whose columns need no padding: a thread owns one unit of one row (two 256-bit
// loads, one 128- or 64-bit code store), the lanes that share a 4-byte scale group merge by shuffle,
// per-thread constants (tensor scale, its reciprocal) are set up once, and a block of 32 x kPairRows
// threads walks row groups with a grid stride so that every SM holds the same amount of work.  Rows
// past data_rows (padding) have zero codes and scales.
//
// The row groups are walked in order, which is also the order of the reduction pass: walked backwards (for
// what the reduction pass left in L2) a static scale pays 0.3 us at 1024 x 3072 (4.72 against 4.43, inputs
// not in L2) and three layers on one 4096 x 3072 input 85.0 against 83.9.  Behind a reduction it pays for fp32 inputs that are larger than
// L2 and marked (walk_of); 16-bit inputs, bound by their arithmetic, gain nothing (36864 x 3072 83.2 / 83.8).
//
// kMark: the input's lines are marked first to leave L2 (evict_first), so that they make room for each other
// and not push out the codes, which the GEMM reads next.  By the rule in walk_of: not for inputs that
// stay in L2, where the next layer on the same activation finds them.
//
// Bound by HBM for large inputs and by launches and latency for small ones: finishing the dynamic scale
// here takes the reduction's last-block tail (and for small inputs the reduction kernel) off the chain.
// Measured, whole calls: 8 x 3072 dynamic linear 39.5 -> 34.8 us; 1003 padded rows through the tensor
// subclass 86.3 -> 70.5 (padded rows took scalar loads before: 6.4 us for 6 MB); an fp32 weight of
// 12288 x 3072 with its dynamic scale 56.8 -> 52.4.
// kPairRows: rows of a thread block, two blocks of 16 to an SM or eight of 4 (launch_streaming_as says when).

template <bool kMark>
__device__ __forceinline__ Vec256 ld_stream_unit(const void* p) {
  if constexpr (kMark) return ld_global_last_use_256(p);
  return ld_global_stream_256(p);
}

template <typename T, bool kHiFirst, bool kDynamic, bool kMark, int kPairRows>
__global__ void __launch_bounds__(32 * kPairRows, 32 / kPairRows)
quantize_nvfp4_stream_kernel(const T* x, const ScaleSource src, uint8_t* __restrict__ codes, uint8_t* __restrict__ scales,
                             int data_rows, int rows, int cols, int rows_pad, int sc_pad, int row_groups) {
  constexpr int kElems = 64 / sizeof(T);  // elements of a thread's unit
  constexpr int kBlocks = kElems / 16;    // scale blocks of a thread's unit
  pdl_launch_dependents();
  const int pc = blockIdx.y * 32 + threadIdx.x;  // unit within the row
  const bool has_data = pc < cols / kElems;
  const bool has_scale = (threadIdx.x & (4 / kBlocks - 1)) == 0 && kBlocks * pc < sc_pad;
  // Ahead of the dependency wait: ask L2 for this block's first two row groups.  A prefetch only
  // warms the cache (L2 is the point of coherence: what the previous kernel still writes is seen
  // by the loads after the wait), and it takes the DRAM latency of the first loads off the
  // critical path of a kernel that only runs for a few microseconds.
  constexpr bool kMayTurn = kDynamic && kMark && sizeof(T) == 4;  // the only form that walk_of sends backwards
  const bool backward = kMayTurn && src.backward;
  const int first = backward ? row_groups - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x);
  const int step = backward ? -static_cast<int>(gridDim.x) : static_cast<int>(gridDim.x);
  if (has_data && (threadIdx.x & 1) == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = (first + i * step) * kPairRows + static_cast<int>(threadIdx.y);
      if ((!kMayTurn || row >= 0) && row < data_rows) prefetch_l2(x + static_cast<int64_t>(row) * cols + pc * kElems);  // one 128-byte line per lane pair
    }
  }
  pdl_wait();  // the tensor scale and x may come from the kernel before this one
  float g;
  if constexpr (kDynamic) {
    // Ahead of the first loads, whose registers would otherwise live across it and spill (44 bytes a thread,
    // two blocks to an SM): one-call linear 65536 x 3072 -> 1024 300 -> 278 us, 12288 x 12288 -> 1024 222 -> 209,
    // the quantizer and its reduction alone 15.0 -> 14.3 at 4096 x 3072, 9.3 -> 8.9 at 2048 x 3072.
    g = block_dynamic_scale(x, src, threadIdx.y * 32 + threadIdx.x, 32 * kPairRows);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) *src.out = g;
  }
  const int col_tiles = sc_pad >> 2;
  const int code_pitch = cols >> 1;
  // The loads of the next row group are issued before the arithmetic of the current one, so
  // memory stays busy while the warps compute.
  Vec256 a = {}, b = {};
  {
    const int row = first * kPairRows + threadIdx.y;
    if (has_data && row < data_rows) {
      const T* at = x + static_cast<int64_t>(row) * cols + pc * kElems;
      a = ld_stream_unit<kMark>(at);
      b = ld_stream_unit<kMark>(at + kElems / 2);
    }
  }
  if constexpr (!kDynamic) g = ld_f32_dependent(src.given);
  const TensorScale ts = make_tensor_scale(g);
  for (int rg = first; (!kMayTurn || rg >= 0) && rg < row_groups; rg += step) {
    const int row = rg * kPairRows + threadIdx.y;
    const int next_row = row + step * kPairRows;
    Vec256 an = {}, bn = {};
    if (has_data && (!kMayTurn || next_row >= 0) && next_row < data_rows) {
      const T* at = x + static_cast<int64_t>(next_row) * cols + pc * kElems;
      an = ld_stream_unit<kMark>(at);
      bn = ld_stream_unit<kMark>(at + kElems / 2);
    }
    uint32_t sb = 0;
    if (has_data && row < rows) {
      uint8_t* const dst = codes + static_cast<int64_t>(row) * code_pitch + pc * (kElems / 2);
      if constexpr (kBlocks == 2) {
        // one block after the other: the straight pair of nvfp4_blocks is slower here (bf16 4096 x 3072 7.3 us against 7.5,
        // 512 x 3072 2.72 against 2.84), where the loads of the next row group are in flight meanwhile
        uint32_t w0, w1, w2, w3, s0, s1;
        nvfp4_block_packed<T, kHiFirst>(a.w, ts, w0, w1, s0);
        nvfp4_block_packed<T, kHiFirst>(b.w, ts, w2, w3, s1);
        *reinterpret_cast<uint4*>(dst) = make_uint4(w0, w1, w2, w3);
        sb = s0 | (s1 << 8);
      } else {
        // fp32: without the two IEEE divisions of a block, 12288 x 3072 with its reduction takes 47.8 us instead of 49.8
        Sixteen<T> x16[1];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          x16[0].w[i] = a.w[i];
          x16[0].w[8 + i] = b.w[i];
        }
        uint32_t out[1][2], scale[1];
        nvfp4_blocks<T, kHiFirst, 1>(x16, ts, out, scale);
        *reinterpret_cast<uint2*>(dst) = make_uint2(out[0][0], out[0][1]);
        sb = scale[0];
      }
    }
    uint32_t word = sb;
    if constexpr (kBlocks == 1) word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1) << 8;
    word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2 / kBlocks) << 16;
    if (has_scale && row < rows_pad) {
      *reinterpret_cast<uint32_t*>(scales + swizzled_scale_offset(row, kBlocks * pc, col_tiles)) = word;
    }
    a = an;
    b = bn;
  }
}

// ---------------------------------------------------------------------------
// MXFP8
// ---------------------------------------------------------------------------
// kVec: whole aligned blocks, unpadded columns.  kPadRows: rows past orig_rows are zeros.
template <typename T, bool kVec, bool kPadRows>
__global__ void __launch_bounds__(kThreads)
quantize_mxfp8_kernel(const T* x, uint8_t* __restrict__ data, uint8_t* __restrict__ scales,
                      int64_t orig_rows, int64_t orig_cols, int64_t num_rows, int64_t num_cols, int64_t sc_pad) {
  pdl_launch_dependents();
  const int64_t sc = blockIdx.y * kColsPerBlock + threadIdx.x;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kRowsPerBlock + threadIdx.y;
  const int64_t n_sc = num_cols >> 5;
  if constexpr (kVec) {
    // ahead of the dependency wait: ask L2 for the thread pair's 128-byte line (warms the cache only)
    if (row < (kPadRows ? orig_rows : num_rows) && sc < n_sc && (threadIdx.x & 1) == 0) prefetch_l2(x + row * orig_cols + sc * 32);
  }
  pdl_wait();
  uint32_t scale_byte = 0;
  if (row < num_rows && sc < n_sc) {
    float lo[16], hi[16];
    if constexpr (kVec && kPadRows) {
#pragma unroll
      for (int i = 0; i < 16; ++i) lo[i] = hi[i] = 0.0f;
      if (row < orig_rows) {
        load16_vec(x + row * orig_cols + sc * 32, lo);
        load16_vec(x + row * orig_cols + sc * 32 + 16, hi);
      }
    } else if constexpr (kVec) {
      load16_vec(x + row * orig_cols + sc * 32, lo);
      load16_vec(x + row * orig_cols + sc * 32 + 16, hi);
    } else {
      load16_guarded(x, row, sc * 32, orig_rows, orig_cols, lo);
      load16_guarded(x, row, sc * 32 + 16, orig_rows, orig_cols, hi);
    }
    const float amax = fmaxf(amax16(lo), amax16(hi));          // :292
    const Mxfp8Scale scale = mxfp8_scale(amax);
    Vec256 out;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      out.w[i] = mxfp8_four(lo + 4 * i, scale);
      out.w[4 + i] = mxfp8_four(hi + 4 * i, scale);
    }
    st_global_256(data + row * num_cols + sc * 32, out);
    scale_byte = scale.byte;
  }
  store_scale_quad(scales, row, sc, sc_pad >> 2, scale_byte, sc < sc_pad);
}

std::atomic<int> g_exact_division{-1};  // -1: not set, follow CK_EXACT_DIV

}  // namespace

bool exact_division() {
  const int v = g_exact_division.load(std::memory_order_relaxed);
  if (v >= 0) return v != 0;
  // CK_EXACT_DIV=1 forces __fdiv_rn for every element (validation of the fast quotient).
  static const bool env = [] {
    const char* e = getenv("CK_EXACT_DIV");
    return e != nullptr && e[0] == '1';
  }();
  return env;
}

namespace {

// The streaming kernel takes rows of whole 64-byte units (rows may be padded, columns not), with
// aligned input and codes.
template <typename T>
bool streaming_applies(const void* input, const void* codes, int64_t orig_rows, int64_t orig_cols, int64_t num_rows, int64_t num_cols) {
  return orig_cols == num_cols && orig_rows <= num_rows && num_cols % (64 / static_cast<int64_t>(sizeof(T))) == 0 &&
         reinterpret_cast<uintptr_t>(input) % 32 == 0 && reinterpret_cast<uintptr_t>(codes) % 16 == 0 &&
         num_rows < (1 << 30) && num_cols < (1 << 30) && !exact_division();
}

// How many passes over the grid a streaming launch makes with all its blocks of 16 rows resident at once.
template <typename T>
int64_t resident_passes(int64_t num_rows, int64_t num_cols) {
  const int64_t col_chunks = ceil_div(round_up(num_cols / 16, 4), 32 * (4 / static_cast<int64_t>(sizeof(T))));
  return ceil_div(round_up(num_rows, 128) / 16 * col_chunks, 2ll * sm_count());
}

// Many passes: blocks of 4 rows that make two each, so that finished blocks make room for the loads of the next.  Graph replays,
// us, resident blocks of 16 rows / so: bf16 8192 x 3072 (6 passes) 13.7 / 14.1, 16384 x 3072 (11) 28.4 / 26.9, 36864 x 3072
// 57.3 / 50.2, fp16 8192 x 15360 54.7 / 51.7, bf16 16384 x 12288 98.8 / 95.5; fp32 12288 x 3072 (16) 25.8 / 27.2, 36864 x 3072
// (47) 90.9 / 78.1.
template <typename T>
bool many_passes(int64_t num_rows, int64_t num_cols) { return resident_passes<T>(num_rows, num_cols) >= (sizeof(T) == 2 ? 8 : 32); }

template <typename T, bool kDynamic, bool kMark, int kPairRows>
int launch_streaming_as(const T* x, const ScaleSource& src, uint8_t* codes, uint8_t* scales, int64_t orig_rows, int64_t num_rows,
                        int64_t num_cols, int hi_first, int most_passes, cudaStream_t stream) {
  const int64_t sc_pad = round_up(num_cols / 16, 4);
  const int rows_pad = static_cast<int>(round_up(num_rows, 128));
  const int row_groups = rows_pad / kPairRows;
  const int col_chunks = static_cast<int>(ceil_div(sc_pad, 32 * (4 / static_cast<int>(sizeof(T)))));
  CK_REQUIRE(col_chunks <= 65535, "quantize_nvfp4: tensor too large for one launch");
  auto kernel = hi_first ? quantize_nvfp4_stream_kernel<T, true, kDynamic, kMark, kPairRows> : quantize_nvfp4_stream_kernel<T, false, kDynamic, kMark, kPairRows>;
  // All blocks resident at once and all of the same length: the grid is the number of
  // row groups divided into the fewest equal passes that fit the device (or into most_passes).
  static std::atomic<int> blocks_per_sm[2] = {{0}, {0}};
  std::atomic<int>& known = blocks_per_sm[hi_first ? 1 : 0];
  int per_sm = known.load(std::memory_order_relaxed);
  if (per_sm == 0) {
    CK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * kPairRows, 0));
    per_sm = max(per_sm, 1);
    known.store(per_sm, std::memory_order_relaxed);
  }
  const int per_wave = max(1, sm_count() * per_sm / col_chunks);
  const int waves = min(static_cast<int>(ceil_div(row_groups, per_wave)), most_passes);
  const int grid_x = static_cast<int>(ceil_div(row_groups, waves));
  const dim3 grid(static_cast<unsigned>(grid_x), static_cast<unsigned>(col_chunks)), block(32, kPairRows);
  CK_CUDA(launch_pdl(kernel, grid, block, 0, stream, x, src, codes, scales, static_cast<int>(orig_rows), static_cast<int>(num_rows),
                     static_cast<int>(num_cols), rows_pad, static_cast<int>(sc_pad), row_groups));
  return CK_OK;
}

template <typename T, bool kMark>
int launch_streaming_marked(const T* x, const ScaleSource& src, uint8_t* codes, uint8_t* scales, int64_t orig_rows, int64_t num_rows,
                            int64_t num_cols, int hi_first, cudaStream_t stream) {
  constexpr int kAll = 1 << 30;
  if (src.given == nullptr) {
    // Every block finishes the scale: few of them.  (One block that finishes it for all, then the launch for many passes:
    // bf16 36864 x 3072 with its reduction 91.0 us instead of 87.9, whose quantizer begins in what the reduction left in L2.)
    return launch_streaming_as<T, true, kMark, 16>(x, src, codes, scales, orig_rows, num_rows, num_cols, hi_first, kAll, stream);
  }
  if (many_passes<T>(num_rows, num_cols)) {
    return launch_streaming_as<T, false, kMark, 4>(x, src, codes, scales, orig_rows, num_rows, num_cols, hi_first, 2, stream);
  }
  // Fewer blocks of 16 rows than SMs: four times as many of 4.  bf16 16 x 3072 2.26 / 1.79 us, 256 x 3072 2.78 / 2.28, 512 x 3072
  // 3.38 / 2.80, 32 x 15360 3.22 / 2.41; with more, 1024 x 3072 3.73 / 3.85, 512 x 15360 6.05 / 6.16.
  const int64_t col_chunks = ceil_div(round_up(num_cols / 16, 4), 32 * (4 / static_cast<int64_t>(sizeof(T))));
  if (round_up(num_rows, 128) / 16 * col_chunks <= sm_count()) {
    return launch_streaming_as<T, false, kMark, 4>(x, src, codes, scales, orig_rows, num_rows, num_cols, hi_first, kAll, stream);
  }
  return launch_streaming_as<T, false, kMark, 16>(x, src, codes, scales, orig_rows, num_rows, num_cols, hi_first, kAll, stream);
}

// How a launch of the streaming quantizer goes through its input.
struct Walk {
  bool mark, backward;
};

// Inputs of more than a quarter of L2 are marked as long as their codes and scales fit in half of it (64 MiB:
// 227 MiB of a 16-bit type, 455 of fp32).  Measured marked / not: three linears on one bf16 activation of
// 24 MiB 91.6 / 89.5 us, of 48 MiB 179.7 / 181.5; fp32 weights of 144 MiB 24.7 / 28.7, of 384 MiB 71.6 / 76.6, of
// 576 MiB 124 / 115; the reduction and quantizer on 384 MiB of bf16 184.8 / 175.4.
//
// Marked fp32 inputs of more than 120 MiB, so up to 455, are quantized from their last rows on, which the reduction has just read.
// Forwards / backwards, us: 6144 x 3072 (72 MiB) 24.1 / 24.3, 8192 x 3072 (96 MiB) 31.4 / 31.6, 12288 x 3072 (144 MiB) 48.0 / 46.4, 24576 x 3072
// 97.6 / 94.7, 36864 x 3072 147 / 143.  Marking what the reduction reads first evict_first, so that the last 64 to 96 MiB stay, gains less
// (47.0 to 47.5 at 144 MiB).
Walk walk_of(int elem_bytes, bool behind_reduction, int64_t orig_rows, int64_t num_rows, int64_t num_cols) {
  const int64_t bytes = orig_rows * num_cols * elem_bytes, written = num_rows * num_cols / 16 * 9;
  Walk w;
  w.mark = bytes > (32ll << 20) && written <= (64ll << 20);
  w.backward = w.mark && behind_reduction && elem_bytes == 4 && bytes > (120ll << 20);
  return w;
}

template <typename T>
int launch_streaming(const T* x, ScaleSource src, uint8_t* codes, uint8_t* scales, int64_t orig_rows, int64_t num_rows,
                     int64_t num_cols, int hi_first, cudaStream_t stream) {
  const Walk walk = walk_of(sizeof(T), src.partials != nullptr, orig_rows, num_rows, num_cols);
  src.backward = walk.backward;
  return walk.mark ? launch_streaming_marked<T, true>(x, src, codes, scales, orig_rows, num_rows, num_cols, hi_first, stream)
                   : launch_streaming_marked<T, false>(x, src, codes, scales, orig_rows, num_rows, num_cols, hi_first, stream);
}

template <typename T>
int launch_nvfp4(const void* input, const float* gs, void* codes, void* scales, int64_t orig_rows, int64_t orig_cols,
                 int64_t num_rows, int64_t num_cols, int hi_first, cudaStream_t stream) {
  const int64_t sc_pad = round_up(num_cols / 16, 4);
  const int64_t grid_rows = round_up(num_rows, 128) / kRowsPerBlock;
  const int64_t grid_cols = ceil_div(sc_pad, kColsPerBlock);
  CK_REQUIRE(grid_rows <= 0x7FFFFFFF && grid_cols <= 65535, "quantize_nvfp4: tensor too large for one launch");
  const T* x = static_cast<const T*>(input);
  uint8_t* c = static_cast<uint8_t*>(codes);
  uint8_t* s = static_cast<uint8_t*>(scales);
  // Small fp32 inputs: the kernel below has twice the blocks of half the threads (not in L2, it / streaming:
  // 128 x 1024 1.69 / 1.85 us, 77 x 4096 2.11 / 2.27, 512 x 1024 1.99 / 2.29; beyond the line 256 x 3072 2.62 / 2.45,
  // 128 x 8192 3.06 / 2.53).  16-bit types and padded rows stream at every size.
  constexpr int64_t kStreamFp32Elements = 640 * 1024;
  const bool small_fp32 = sizeof(T) == 4 && orig_rows == num_rows && round_up(num_rows, 128) * num_cols < kStreamFp32Elements;
  if (!small_fp32 && streaming_applies<T>(input, codes, orig_rows, orig_cols, num_rows, num_cols)) {
    ScaleSource src = {};
    src.given = gs;
    return launch_streaming<T>(x, src, c, s, orig_rows, num_rows, num_cols, hi_first, stream);
  }
  const dim3 grid(static_cast<unsigned>(grid_rows), static_cast<unsigned>(grid_cols)), block(kColsPerBlock, kRowsPerBlock);
  // vector path: every 16-element run is inside the input and 32-byte aligned
  const bool vec = (orig_rows == num_rows) && (orig_cols == num_cols) &&
                   (reinterpret_cast<uintptr_t>(input) % 32 == 0);
  const bool exact = exact_division();
#define CK_LAUNCH(VEC, FAST)                                                                                  \
  CK_CUDA(launch_pdl(quantize_nvfp4_kernel<T, VEC, FAST>, grid, block, 0, stream, x, gs, c, s, orig_rows, orig_cols, \
                     num_rows, num_cols, sc_pad, hi_first))
  if (vec) {
    if (exact) CK_LAUNCH(true, false); else CK_LAUNCH(true, true);
  } else {
    if (exact) CK_LAUNCH(false, false); else CK_LAUNCH(false, true);
  }
#undef CK_LAUNCH
  CK_CUDA(cudaGetLastError());
  return CK_OK;
}

// Inputs of at most this many bytes: every block of the quantizer takes the maximum of the whole input
// itself (a few 16 KiB passes out of L2) instead of waiting for a reduction kernel, which is a launch more.  Scale and quantizer, us, reduction
// kernel / whole input: bf16 16 x 3072 (96 KiB) 4.1 / 3.4, 22 x 3072 (132 KiB) 4.0 / 3.5, 32 x 3072 (192 KiB) 4.1 / 4.1, 40 x 3072 4.1 / 4.8, fp16 64
// x 1024 (128 KiB) 3.9 / 3.3, fp32 12 x 3072 (144 KiB) 3.4 / 3.5; linears bf16 12 x 3072 x 3072 9.0 / 8.1, 9 x 9216 x 5120 11.7 / 10.8, 12 x 3072 x
// 6144 (144 KiB) 9.1 / 9.5, 64 x 9216 x 1024 8.2 / 7.4.  Up to eight rows, whose quantizer blocks are narrow and many, the line stays lower: 8 x 4096
// (64 KiB) 4.4 / 3.5, 3 x 15360 (90 KiB) 3.6 / 3.8, 8 x 15360 4.0 / 5.6.
constexpr int64_t whole_input_bytes(int64_t rows) { return rows > 8 ? 128 * 1024 : 64 * 1024; }
constexpr int64_t kDynamicScratchHead = 256;

__global__ void clear_word_kernel(unsigned int* word) {
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) *word = 0;
}

template <typename T>
int launch_nvfp4_dynamic(const void* input, int dtype, float* scale_out, void* codes, void* scales, int64_t orig_rows,
                         int64_t orig_cols, int64_t num_rows, int64_t num_cols, int hi_first, void* scratch,
                         int64_t scratch_bytes, cudaStream_t stream) {
  const int64_t n = orig_rows * orig_cols;
  if (streaming_applies<T>(input, codes, orig_rows, orig_cols, num_rows, num_cols)) {
    const T* x = static_cast<const T*>(input);
    ScaleSource src = {};
    src.out = scale_out;
    src.n_vecs = n / (32 / static_cast<int64_t>(sizeof(T)));
    if (n * static_cast<int64_t>(sizeof(T)) > whole_input_bytes(orig_rows)) {
      // behind the arrival counter of the one-kernel reduction, which may share this scratch and wants it zero
      float* partials = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kDynamicScratchHead);
      if (int rc = launch_amax_partials(x, dtype, src.n_vecs, partials, &src.n_partials, stream)) return rc;
      src.partials = partials;
    }
    return launch_streaming<T>(x, src, static_cast<uint8_t*>(codes), static_cast<uint8_t*>(scales), orig_rows, num_rows, num_cols,
                               hi_first, stream);
  }
  // The one-kernel reduction keeps an arrival counter at the head of its scratch, which has to start at zero: cleared
  // by a kernel, since a memset node would break the chain of dependent launches (8 x 3072 off by one element:
  // 11.6 us with it, 8.3 so, 7.6 for the two calls on a scratch that is zero).
  CK_CUDA(launch_pdl(clear_word_kernel, dim3(1), dim3(32), 0, stream, static_cast<unsigned int*>(scratch)));
  if (int rc = ck_nvfp4_tensor_scale(input, dtype, n, scale_out, scratch, scratch_bytes, stream)) return rc;
  return launch_nvfp4<T>(input, scale_out, codes, scales, orig_rows, orig_cols, num_rows, num_cols, hi_first, stream);
}

template <typename T>
int launch_mxfp8(const void* input, void* data, void* scales, int64_t orig_rows, int64_t orig_cols, int64_t num_rows,
                 int64_t num_cols, cudaStream_t stream) {
  const int64_t sc_pad = round_up(num_cols / 32, 4);
  const int64_t grid_rows = round_up(num_rows, 128) / kRowsPerBlock;
  const int64_t grid_cols = ceil_div(sc_pad, kColsPerBlock);
  CK_REQUIRE(grid_rows <= 0x7FFFFFFF && grid_cols <= 65535, "quantize_mxfp8: tensor too large for one launch");
  const dim3 grid(static_cast<unsigned>(grid_rows), static_cast<unsigned>(grid_cols)), block(kColsPerBlock, kRowsPerBlock);
  const bool vec = (orig_cols == num_cols) &&
                   (reinterpret_cast<uintptr_t>(input) % 32 == 0) && (reinterpret_cast<uintptr_t>(data) % 32 == 0);
  const T* x = static_cast<const T*>(input);
  uint8_t* d = static_cast<uint8_t*>(data);
  uint8_t* s = static_cast<uint8_t*>(scales);
  if (vec) {
    // Without rows to pad, 16-bit types take the loads without the select (not in L2, without / with: bf16
    // 4096 x 3072 6.39 / 6.57 us, 1024 x 3072 2.94 / 3.05, 36864 x 3072 53.7 / 54.5); fp32 is faster with it (4096 x 3072
    // 10.35 / 10.40, 12288 x 3072 31.0 / 30.6, 16384 x 12288 163.0 / 159.9).
    constexpr bool kFp32 = sizeof(T) == 4;
    auto kernel = orig_rows == num_rows ? quantize_mxfp8_kernel<T, true, kFp32> : quantize_mxfp8_kernel<T, true, true>;
    CK_CUDA(launch_pdl(kernel, grid, block, 0, stream, x, d, s, orig_rows, orig_cols, num_rows, num_cols, sc_pad));
  } else {
    CK_REQUIRE(reinterpret_cast<uintptr_t>(data) % 32 == 0, "quantize_mxfp8: output must be 32-byte aligned");
    CK_CUDA(launch_pdl(quantize_mxfp8_kernel<T, false, true>, grid, block, 0, stream, x, d, s, orig_rows, orig_cols, num_rows,
                       num_cols, sc_pad));
  }
  CK_CUDA(cudaGetLastError());
  return CK_OK;
}

int check_quant_shapes(const char* op, int64_t block, const void* input, const void* out, const void* scales,
                       int64_t orig_rows, int64_t orig_cols, int64_t num_rows, int64_t num_cols) {
  CK_REQUIRE(input && out && scales, "%s: null pointer", op);
  CK_REQUIRE(orig_rows > 0 && orig_cols > 0, "%s: empty input [%lld, %lld]", op, (long long)orig_rows,
             (long long)orig_cols);
  CK_REQUIRE(num_cols % block == 0, "%s: num_cols=%lld is not a multiple of %lld", op, (long long)num_cols,
             (long long)block);
  const bool same = (num_rows == orig_rows && num_cols == orig_cols);
  const bool padded = (num_rows == round_up(orig_rows, block) && num_cols == round_up(orig_cols, block));
  CK_REQUIRE(same || padded, "%s: output [%lld, %lld] is neither the input shape [%lld, %lld] nor its %lld-padding",
             op, (long long)num_rows, (long long)num_cols, (long long)orig_rows, (long long)orig_cols,
             (long long)block);
  CK_REQUIRE(reinterpret_cast<uintptr_t>(scales) % 4 == 0, "%s: block_scales must be 4-byte aligned", op);
  return CK_OK;
}

}  // namespace
}  // namespace ck

extern "C" int ck_debug_set_exact_division(int on) {
  const bool before = ck::exact_division();
  ck::g_exact_division.store(on != 0 ? 1 : 0, std::memory_order_relaxed);
  return before ? 1 : 0;
}

extern "C" int ck_debug_quantize_nvfp4_walk(int input_dtype, int dynamic, int64_t rows, int64_t cols) {
  const bool fp32 = input_dtype == CK_DTYPE_F32;
  const int elem = fp32 ? 4 : 2;
  const ck::Walk w = ck::walk_of(elem, dynamic != 0 && rows * cols * elem > ck::whole_input_bytes(rows), rows, rows, cols);
  return (w.mark ? 1 : 0) | (w.backward ? 2 : 0);
}

extern "C" int ck_quantize_nvfp4(const void* input, int input_dtype, const float* global_scale, void* codes,
                                 void* block_scales, int64_t orig_rows, int64_t orig_cols, int64_t num_rows,
                                 int64_t num_cols, int hi_first, void* stream) {
  using namespace ck;
  if (int rc = check_quant_shapes("quantize_nvfp4", 16, input, codes, block_scales, orig_rows, orig_cols, num_rows,
                                  num_cols))
    return rc;
  CK_REQUIRE(global_scale != nullptr, "quantize_nvfp4: null global_scale");
  CK_REQUIRE(reinterpret_cast<uintptr_t>(codes) % 8 == 0, "quantize_nvfp4: codes must be 8-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (input_dtype) {
    case CK_DTYPE_BF16:
      return launch_nvfp4<__nv_bfloat16>(input, global_scale, codes, block_scales, orig_rows, orig_cols, num_rows,
                                         num_cols, hi_first, s);
    case CK_DTYPE_F16:
      return launch_nvfp4<__half>(input, global_scale, codes, block_scales, orig_rows, orig_cols, num_rows, num_cols,
                                  hi_first, s);
    case CK_DTYPE_F32:
      return launch_nvfp4<float>(input, global_scale, codes, block_scales, orig_rows, orig_cols, num_rows, num_cols,
                                 hi_first, s);
    default:
      return fail(CK_ERR_INVALID_ARGUMENT, "quantize_nvfp4: unsupported input dtype code %d", input_dtype);
  }
}

extern "C" int64_t ck_quantize_nvfp4_dynamic_scratch_bytes(int64_t num_elements) {
  if (num_elements <= 0) return 0;
  // the most of all types (fp32 has eight elements to a 32-byte unit) and of both routes
  const int64_t partials = ck::kDynamicScratchHead + 4 * ck::amax_partials(ck::ceil_div(num_elements, 8));
  const int64_t general = ck_nvfp4_tensor_scale_scratch_bytes(num_elements);
  return general > partials ? general : partials;
}

extern "C" int64_t ck_quantize_nvfp4_dynamic_whole_input_bytes(int64_t orig_rows) { return ck::whole_input_bytes(orig_rows); }

extern "C" int ck_quantize_nvfp4_dynamic(const void* input, int input_dtype, float* scale_out, void* codes, void* block_scales,
                                         int64_t orig_rows, int64_t orig_cols, int64_t num_rows, int64_t num_cols, int hi_first,
                                         void* scratch, int64_t scratch_bytes, void* stream) {
  using namespace ck;
  if (int rc = check_quant_shapes("quantize_nvfp4_dynamic", 16, input, codes, block_scales, orig_rows, orig_cols, num_rows, num_cols))
    return rc;
  CK_REQUIRE(scale_out != nullptr && scratch != nullptr, "quantize_nvfp4_dynamic: null scale_out or scratch");
  CK_REQUIRE(reinterpret_cast<uintptr_t>(codes) % 8 == 0, "quantize_nvfp4_dynamic: codes must be 8-byte aligned");
  CK_REQUIRE(reinterpret_cast<uintptr_t>(scratch) % 4 == 0 && scratch_bytes >= ck_quantize_nvfp4_dynamic_scratch_bytes(orig_rows * orig_cols),
             "quantize_nvfp4_dynamic: scratch of %lld bytes, %lld needed (4-byte aligned)", (long long)scratch_bytes,
             (long long)ck_quantize_nvfp4_dynamic_scratch_bytes(orig_rows * orig_cols));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (input_dtype) {
    case CK_DTYPE_BF16:
      return launch_nvfp4_dynamic<__nv_bfloat16>(input, input_dtype, scale_out, codes, block_scales, orig_rows, orig_cols, num_rows,
                                                 num_cols, hi_first, scratch, scratch_bytes, s);
    case CK_DTYPE_F16:
      return launch_nvfp4_dynamic<__half>(input, input_dtype, scale_out, codes, block_scales, orig_rows, orig_cols, num_rows, num_cols,
                                          hi_first, scratch, scratch_bytes, s);
    case CK_DTYPE_F32:
      return launch_nvfp4_dynamic<float>(input, input_dtype, scale_out, codes, block_scales, orig_rows, orig_cols, num_rows, num_cols,
                                         hi_first, scratch, scratch_bytes, s);
    default:
      return fail(CK_ERR_INVALID_ARGUMENT, "quantize_nvfp4_dynamic: unsupported input dtype code %d", input_dtype);
  }
}

extern "C" int ck_quantize_mxfp8(const void* input, int input_dtype, void* data, void* block_scales,
                                 int64_t orig_rows, int64_t orig_cols, int64_t num_rows, int64_t num_cols,
                                 void* stream) {
  using namespace ck;
  if (int rc = check_quant_shapes("quantize_mxfp8", 32, input, data, block_scales, orig_rows, orig_cols, num_rows,
                                  num_cols))
    return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (input_dtype) {
    case CK_DTYPE_BF16:
      return launch_mxfp8<__nv_bfloat16>(input, data, block_scales, orig_rows, orig_cols, num_rows, num_cols, s);
    case CK_DTYPE_F16:
      return launch_mxfp8<__half>(input, data, block_scales, orig_rows, orig_cols, num_rows, num_cols, s);
    case CK_DTYPE_F32:
      return launch_mxfp8<float>(input, data, block_scales, orig_rows, orig_cols, num_rows, num_cols, s);
    default:
      return fail(CK_ERR_INVALID_ARGUMENT, "quantize_mxfp8: unsupported input dtype code %d", input_dtype);
  }
}
