// Host-side helpers shared by the TMA kernels: encode tensor maps (128-byte swizzle)
// through the driver entry point, resolved at run time so the library has no link-time
// dependency on libcuda.
#pragma once
#include "common.cuh"
#include <cuda.h>
#include <stdio.h>

namespace bbhost {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(sym);
  return fn;
}

// The driver call needs a context bound to the calling thread; a thread that has only ever
// set its device (autograd worker threads) has none yet.
inline int bind_context() {
  static thread_local bool bound = false;
  if (!bound) {
    cudaError_t e = cudaFree(0);
    if (e != cudaSuccess) { bb_set_last_error("cudaFree(0)", e); return BB_ERR_CUDA; }
    bound = true;
  }
  return BB_OK;
}

// Tensor map of `rank` dimensions (innermost first, 128-byte swizzle unless named) over bf16, or fp32 when f32 != 0; `pitch`: bytes
// between neighbours of every dimension but the innermost.
inline int encode_tiled(CUtensorMap* tm, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* pitch,
                        const cuuint32_t* box, int f32, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) { bb_set_last_error_msg("cuTensorMapEncodeTiled entry point not available"); return BB_ERR_CUDA; }
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(tm, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base),
                  dims, pitch, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char msg[256];
    snprintf(msg, sizeof(msg), "cuTensorMapEncodeTiled failed with CUresult %d (base %p, rows %lld, cols %lld, row pitch %lld bytes, box %ux%u, "
             "f32 %d); operands need a 16-byte aligned base and row pitch", (int)r, base, (long long)dims[1], (long long)dims[0],
             (long long)pitch[0], box[0], box[1], f32);
    bb_set_last_error_msg(msg);
    return BB_ERR_INVALID_ARG;
  }
  return BB_OK;
}

// 2-D tensor map over a row-major [rows, cols] matrix with leading dimension ld (elements); box = box_cols x box_rows.
inline int encode_2d(CUtensorMap* tm, const void* base, long long rows, long long cols, long long ld, int box_cols, int box_rows,
                     int f32 = 0, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, pitch[1] = {(cuuint64_t)ld * (f32 ? 4 : 2)};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  return encode_tiled(tm, base, 2, dims, pitch, box, f32, swizzle);
}

// 3-D tensor map over `seqs` sequences of `rows` bf16 rows each, one after the other in a [seqs * rows, cols] matrix.  A box
// ends with its sequence: rows past the end load as zeros.
inline int encode_seqs(CUtensorMap* tm, const void* base, int seqs, int rows, long long cols, long long ld, int box_cols, int box_rows) {
  const cuuint64_t row = (cuuint64_t)ld * 2;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)seqs}, pitch[2] = {row, row * (cuuint64_t)rows};
  const cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1};
  return encode_tiled(tm, base, 3, dims, pitch, box, 0);
}

typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const int*, const int*, cuuint32_t, cuuint32_t, const cuuint32_t*,
                                   CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// im2col tensor map over an NHWC bf16 tensor: `pixels` consecutive output positions of a k x k window with the
// given stride and padding, 64 channels each (128-byte swizzle).  The windows' first taps run over
// [-pad, size + pad - k] in steps of `stride`; a tap is chosen per load by its offset.
inline int encode_im2col(CUtensorMap* tm, const void* base, int N, int H, int W, int C, int k, int stride, int pad, int pixels) {
  static EncodeIm2colFn fn = nullptr;
  if (!fn) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &sym, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess) {
      bb_set_last_error_msg("cuTensorMapEncodeIm2col entry point not available");
      return BB_ERR_CUDA;
    }
    fn = reinterpret_cast<EncodeIm2colFn>(sym);
  }
  cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
  cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
  int lower[2] = {-pad, -pad}, upper[2] = {pad - (k - 1), pad - (k - 1)};
  cuuint32_t estr[4] = {1, (cuuint32_t)stride, (cuuint32_t)stride, 1};
  CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, lower, upper, 64, (cuuint32_t)pixels,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char msg[256];
    snprintf(msg, sizeof(msg), "cuTensorMapEncodeIm2col failed with CUresult %d (base %p, NHWC %d x %d x %d x %d, k %d, stride %d, pad %d)",
             (int)r, base, N, H, W, C, k, stride, pad);
    bb_set_last_error_msg(msg);
    return BB_ERR_INVALID_ARG;
  }
  return BB_OK;
}

}  // namespace bbhost
