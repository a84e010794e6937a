// Dequantizers for sm_100a: NVFP4 (packed E2M1 + tiled E4M3 scales + fp32 tensor scale) and
// MXFP8 (E4M3 + tiled E8M0 scales) back to f32 / f16 / bf16.  Streaming kernels bounded by
// the output write: one thread per scale block, 256-bit stores.
//
// Arithmetic contract (bit-identical to the reference's eager path):
//   NVFP4, comfy_kitchen/backends/eager/quantization.py:171-219: everything happens in the
//     OUTPUT dtype: total = out_t(tensor_scale) * out_t(block_scale), value = lut * total.
//   MXFP8, :327-364: float32(e4m3) * 2^(e-127) in float32 (scale byte 0 decodes to 0), then
//     one cast to the output dtype.
#include "ck_common.cuh"

#include <type_traits>

namespace ck {
namespace {

constexpr int kThreads = 256;

template <typename OutT>
__device__ __forceinline__ float round_to(float v) {
  if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
    return __bfloat162float(__float2bfloat16_rn(v));
  } else if constexpr (std::is_same<OutT, __half>::value) {
    return __half2float(__float2half_rn(v));
  } else {
    return v;
  }
}

template <typename OutT>
__device__ __forceinline__ void store16(OutT* dst, const float (&v)[16]) {
  if constexpr (sizeof(OutT) == 2) {
    Vec256 o;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
        __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        o.w[i] = *reinterpret_cast<uint32_t*>(&p);
      } else {
        __half2 p = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
        o.w[i] = *reinterpret_cast<uint32_t*>(&p);
      }
    }
    st_global_256(dst, o);
  } else {
    Vec256 a, b;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a.w[i] = __float_as_uint(v[i]);
      b.w[i] = __float_as_uint(v[8 + i]);
    }
    st_global_256(dst, a);
    st_global_256(dst + 8, b);
  }
}

__device__ __forceinline__ float e4m3_byte_to_f32(uint32_t b) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<uint16_t>(b)));
  return __half2float(__ushort_as_half(static_cast<unsigned short>(h2 & 0xFFFFu)));
}

// Four packed bytes (eight E2M1 codes) -> four f16x2 pairs with the hardware convert; in each
// pair the low half comes from the low nibble of its byte.  Every E2M1 value is exact in f16.
__device__ __forceinline__ void e2m1x8_to_f16x2(uint32_t word, uint32_t (&h)[4]) {
  asm("{ .reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3; }"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(word));
}

// Bound by HBM (the result's write) for large tensors, by launch and latency for small ones.  A thread takes a 16- (NVFP4) or
// 32-element (MXFP8) block of one row, or of two, four apart (kRows, NVFP4).  Launched like the other streaming kernels, as a dependent of
// the kernel before it.
//
// `early`: whether the next kernel's blocks may come once this block's loads are under way (else with its end).  Up to there a block
// waits for the kernel before it, so that no third kernel gets in: blocks of several launches that wait together leave the next
// launch a few SMs, where they bunch.  Triggered first thing, the back-to-back calls that now take 2.9 us (MXFP8 to fp32, 500 x 2816) took
// 6.4, launched plainly 3.1.  Not where fp32 results of one to six (MXFP8: ten) blocks an SM keep the memory busy by themselves.  Graph replays,
// us, launched plainly / triggered first thing / early / not: NVFP4 to bf16 300 x 768 1.65 / 1.33 / 1.11 / 1.30, 1200 x 2816 3.34 / 2.67 / 2.62 / 3.02, MXFP8 to
// bf16 500 x 2816 2.59 / 3.08 / 2.21 / 2.48, 800 x 4480 3.49 / 3.67 / 3.00 / 3.37; to fp32, up to 148 blocks: NVFP4 300 x 768 2.13 / 1.71 / 1.56 / 2.02,
// MXFP8 128 x 4480 3.00 / 4.97 / 2.59 / 2.83; more: NVFP4 800 x 2816 2.94 / 3.26 / 3.46 / 2.74, MXFP8 300 x 12288 6.43 / 9.00 / 7.63 / 5.94, 1658 x 4480
// 10.04 / 10.74 / 10.48 / 9.63; beyond: NVFP4 800 x 4480 4.11 / 3.98 / 3.98 / 4.10, 2400 x 2816 6.93 / 6.37 / 6.34 / 6.67, MXFP8 6000 x 768 7.20 / 7.05 / 6.59 / 7.04.
//
// Two rows in flight pay where a thread's traffic is small, for NVFP4 to a 16-bit type, and where the blocks of one row do not all fit
// at once (eight to an SM, 1184: 4.85 million elements).  One row / two, us, bf16: 1365 x 3072 (1026 blocks) 2.88 / 3.38, 4736 x 1024 (1184)
// 3.03 / 3.55, 5000 x 1024 (1250) 3.94 / 3.68, 1600 x 3072 (1200) 3.86 / 3.68, 12288 x 3072 17.98 / 16.87; four 17.5.  To fp32 4096 x 3072 10.7 / 10.6 / 11.7;
// MXFP8 to bf16 12288 x 3072 18.8 / 19.2 / 20.2.
template <typename OutT, bool kHiFirst, int kRows>
__global__ void __launch_bounds__(kThreads)
dequantize_nvfp4_kernel(const uint8_t* codes, const float* global_scale, const uint8_t* scales, OutT* __restrict__ out, int64_t rows, int64_t cols,
                        bool early) {
  const int64_t n_sc = cols >> 4;
  const int64_t sc = static_cast<int64_t>(blockIdx.y) * 64 + threadIdx.x;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * (4 * kRows) + threadIdx.y;
  const int64_t col_tiles = ceil_div(n_sc, 4);
  if constexpr (kRows == 1) {
    // ahead of the dependency wait: ask L2 for the 128-byte line of sixteen threads (warms the cache only)
    if (sc < n_sc && row0 < rows && (threadIdx.x & 15) == 0) prefetch_l2(codes + row0 * (cols >> 1) + sc * 8);
  }
  pdl_wait();
  if (sc >= n_sc) return;
  uint2 packed[kRows];
  uint32_t sbyte[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int64_t row = row0 + 4 * i;
    if (row < rows) {
      packed[i] = ld_global_stream_64(codes + row * (cols >> 1) + sc * 8);
      sbyte[i] = ld_global_u8(scales + swizzled_scale_offset(row, sc, col_tiles));
    }
  }
  if (early) pdl_launch_dependents();
  // :211 total scale in the output dtype
  const float ts = round_to<OutT>(ld_f32_dependent(global_scale));
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int64_t row = row0 + 4 * i;
    if (row >= rows) break;
    const float bs = e4m3_byte_to_f32(sbyte[i]);  // exact in every output dtype
    const float total = round_to<OutT>(ts * bs);
    float v[16];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      uint32_t h[4];
      e2m1x8_to_f16x2(w == 0 ? packed[i].x : packed[i].y, h);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[j]));  // (low nibble, high nibble)
        // :214, rounded by the store; the product of two OutT numbers is exact in float32
        v[8 * w + 2 * j] = (kHiFirst ? f.y : f.x) * total;
        v[8 * w + 2 * j + 1] = (kHiFirst ? f.x : f.y) * total;
      }
    }
    store16<OutT>(out + row * cols + sc * 16, v);
  }
}

template <typename OutT>
__global__ void __launch_bounds__(kThreads)
dequantize_mxfp8_kernel(const uint8_t* data, const uint8_t* scales, OutT* __restrict__ out, int64_t rows, int64_t cols, bool early) {
  const int64_t n_sc = cols >> 5;
  const int64_t sc = static_cast<int64_t>(blockIdx.y) * 64 + threadIdx.x;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * 4 + threadIdx.y;
  pdl_wait();
  if (row >= rows || sc >= n_sc) return;
  const Vec256 raw = ld_global_stream_256(data + row * cols + sc * 32);
  const uint32_t e = ld_global_u8(scales + swizzled_scale_offset(row, sc, ceil_div(n_sc, 4)));
  if (early) pdl_launch_dependents();
  const float scale = __uint_as_float(e << 23);  // byte 0 -> 0.0 (float_utils.py:376-382)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float v[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w = raw.w[h * 4 + j];
      v[4 * j + 0] = e4m3_byte_to_f32(w & 0xFFu) * scale;
      v[4 * j + 1] = e4m3_byte_to_f32((w >> 8) & 0xFFu) * scale;
      v[4 * j + 2] = e4m3_byte_to_f32((w >> 16) & 0xFFu) * scale;
      v[4 * j + 3] = e4m3_byte_to_f32(w >> 24) * scale;
    }
    store16<OutT>(out + row * cols + sc * 32 + h * 16, v);
  }
}

int check_common(const char* op, const void* in, const void* scales, const void* out, int out_dtype, int64_t rows,
                 int64_t cols, int64_t block) {
  CK_REQUIRE(in && scales && out, "%s: null pointer", op);
  CK_REQUIRE(rows > 0 && cols > 0 && cols % block == 0, "%s: bad shape [%lld, %lld]", op, (long long)rows,
             (long long)cols);
  CK_REQUIRE(out_dtype == CK_DTYPE_F32 || out_dtype == CK_DTYPE_F16 || out_dtype == CK_DTYPE_BF16,
             "%s: unsupported output dtype code %d", op, out_dtype);
  CK_REQUIRE(reinterpret_cast<uintptr_t>(out) % 32 == 0, "%s: output must be 32-byte aligned", op);
  CK_REQUIRE(ceil_div(rows, 4) <= 0x7FFFFFFF && ceil_div(cols / block, 64) <= 65535, "%s: tensor too large", op);
  return CK_OK;
}

// See above the kernels.
template <typename OutT>
bool triggers_early(const dim3& grid, int many_to_an_sm) {
  const int64_t blocks = static_cast<int64_t>(grid.x) * grid.y;
  return sizeof(OutT) == 2 || blocks <= sm_count() || blocks > static_cast<int64_t>(many_to_an_sm) * sm_count();
}

template <typename OutT, int kRows>
int launch_nvfp4_rows(const uint8_t* codes, const float* global_scale, const uint8_t* scales, void* out, int64_t rows, int64_t cols, int hi_first,
                      cudaStream_t stream) {
  const dim3 grid(static_cast<unsigned>(ceil_div(rows, 4 * kRows)), static_cast<unsigned>(ceil_div(cols / 16, 64))), block(64, 4);
  auto kernel = hi_first ? dequantize_nvfp4_kernel<OutT, true, kRows> : dequantize_nvfp4_kernel<OutT, false, kRows>;
  CK_CUDA(launch_pdl(kernel, grid, block, 0, stream, codes, global_scale, scales, static_cast<OutT*>(out), rows, cols,
                     triggers_early<OutT>(grid, 6)));
  return CK_OK;
}

template <typename OutT>
int launch_nvfp4(const uint8_t* codes, const float* global_scale, const uint8_t* scales, void* out, int64_t rows, int64_t cols, int hi_first,
                 cudaStream_t stream) {
  if constexpr (sizeof(OutT) == 2) {
    constexpr int64_t kBlocksPerSm = 2048 / kThreads;
    if (ceil_div(rows, 4) * ceil_div(cols / 16, 64) > kBlocksPerSm * sm_count()) {
      return launch_nvfp4_rows<OutT, 2>(codes, global_scale, scales, out, rows, cols, hi_first, stream);
    }
  }
  return launch_nvfp4_rows<OutT, 1>(codes, global_scale, scales, out, rows, cols, hi_first, stream);
}

template <typename OutT>
int launch_mxfp8(const uint8_t* data, const uint8_t* scales, void* out, int64_t rows, int64_t cols, cudaStream_t stream) {
  const dim3 grid(static_cast<unsigned>(ceil_div(rows, 4)), static_cast<unsigned>(ceil_div(cols / 32, 64))), block(64, 4);
  CK_CUDA(launch_pdl(dequantize_mxfp8_kernel<OutT>, grid, block, 0, stream, data, scales, static_cast<OutT*>(out), rows, cols,
                     triggers_early<OutT>(grid, 10)));
  return CK_OK;
}

}  // namespace
}  // namespace ck

extern "C" int ck_dequantize_nvfp4(const void* codes, const float* global_scale, const void* block_scales, void* out,
                                   int out_dtype, int64_t rows, int64_t cols, int hi_first, void* stream) {
  using namespace ck;
  if (int rc = check_common("dequantize_nvfp4", codes, block_scales, out, out_dtype, rows, cols, 16)) return rc;
  CK_REQUIRE(global_scale != nullptr, "dequantize_nvfp4: null global_scale");
  CK_REQUIRE(reinterpret_cast<uintptr_t>(codes) % 8 == 0, "dequantize_nvfp4: codes must be 8-byte aligned");
  const uint8_t* c = static_cast<const uint8_t*>(codes);
  const uint8_t* sc = static_cast<const uint8_t*>(block_scales);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (out_dtype) {
    case CK_DTYPE_BF16: return launch_nvfp4<__nv_bfloat16>(c, global_scale, sc, out, rows, cols, hi_first, s);
    case CK_DTYPE_F16: return launch_nvfp4<__half>(c, global_scale, sc, out, rows, cols, hi_first, s);
    default: return launch_nvfp4<float>(c, global_scale, sc, out, rows, cols, hi_first, s);
  }
}

extern "C" int ck_dequantize_mxfp8(const void* data, const void* block_scales, void* out, int out_dtype, int64_t rows,
                                   int64_t cols, void* stream) {
  using namespace ck;
  if (int rc = check_common("dequantize_mxfp8", data, block_scales, out, out_dtype, rows, cols, 32)) return rc;
  CK_REQUIRE(reinterpret_cast<uintptr_t>(data) % 32 == 0, "dequantize_mxfp8: data must be 32-byte aligned");
  const uint8_t* d = static_cast<const uint8_t*>(data);
  const uint8_t* sc = static_cast<const uint8_t*>(block_scales);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (out_dtype) {
    case CK_DTYPE_BF16: return launch_mxfp8<__nv_bfloat16>(d, sc, out, rows, cols, s);
    case CK_DTYPE_F16: return launch_mxfp8<__half>(d, sc, out, rows, cols, s);
    default: return launch_mxfp8<float>(d, sc, out, rows, cols, s);
  }
}
