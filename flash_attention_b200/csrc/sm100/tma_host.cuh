// Host-side construction of TMA tensor maps for (batch, seq, head, dim) operands with arbitrary
// 16-byte-aligned strides.  The driver entry point is resolved at run time so that the library
// links against the CUDA runtime only.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../fa_common.cuh"

namespace fa {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn encode_tiled_fn() {
  // (looked up once, by the first of several threads: whether it is there decides which kernel a plan and its call choose)
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeTiledFn>(p);
    cudaGetLastError();
    return nullptr;
  }();
  return fn;
}

static inline int make_tmap(CUtensorMap* map, const FaTensor& t, int dtype, int head_dim, const int64_t (&extent)[3],
                            const int64_t (&stride)[3], const int (&box_of)[3]) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) {
    fa_host::set_error("cuTensorMapEncodeTiled is not available from this driver");
    return 1;
  }
  cuuint64_t dims[4] = {(cuuint64_t)head_dim, (cuuint64_t)extent[0], (cuuint64_t)extent[1], (cuuint64_t)extent[2]};
  // strides of dims 1..3 in bytes; a dim of one element still needs a legal (non-zero, 16 B multiple) stride, whatever it
  // is.  (A stride of 0 on more elements does not come here: tma_compatible refuses it.)
  auto legal = [](int64_t elems) { return (cuuint64_t)(elems > 0 ? elems : 8) * 2; };
  cuuint64_t strides[3] = {legal(stride[0]), legal(stride[1]), legal(stride[2])};
  cuuint32_t box[4] = {64, (cuuint32_t)box_of[0], (cuuint32_t)box_of[1], (cuuint32_t)box_of[2]};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  auto encode = [&]() { return fn(map, dtype == FA_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                  t.ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE); };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {  // a thread that has made no runtime call yet (autograd's): make its context current
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
  }
  if (r != CUDA_SUCCESS) {
    fa_host::set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return 1;
  }
  return 0;
}

// 4-D map with dims (dim, seq, head, batch), 128-byte swizzle, box = 64 elements x box_rows rows.
// Out-of-range elements read as zero.  `rows`/`batches` describe the extent of the tensor: for
// packed variable-length tensors rows = total tokens and batches = 1.
static inline int make_tmap_4d(CUtensorMap* map, const FaTensor& t, int dtype, int64_t rows, int heads, int64_t batches,
                               int head_dim, int box_rows) {
  return make_tmap(map, t, dtype, head_dim, {rows, heads, batches}, {t.stride_s, t.stride_h, t.stride_b}, {box_rows, 1, 1});
}

// The same tensor with dims (dim, head, seq, batch) and a box of box_heads heads of box_rows positions: the rows of a
// box are ordered (position, head).
static inline int make_tmap_4d_heads(CUtensorMap* map, const FaTensor& t, int dtype, int64_t rows, int heads, int64_t batches,
                                     int head_dim, int box_heads, int box_rows) {
  return make_tmap(map, t, dtype, head_dim, {heads, rows, batches}, {t.stride_h, t.stride_s, t.stride_b},
                   {box_heads, box_rows, 1});
}

// Base and strides in 16-byte pieces
static inline bool rows_compatible(const FaTensor& t) {
  auto ok = [](int64_t s) { return s >= 0 && s % 8 == 0 && s < (1ll << 38); };
  return (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && ok(t.stride_s) && ok(t.stride_h) && ok(t.stride_b);
}

// ... and no dim that repeats its elements: a map has no stride of 0, the kernels that take addresses do.  (A null pointer
// is a plan made before the tensors exist: its strides say nothing yet.)
static inline bool tma_compatible(const FaTensor& t, int64_t rows, int64_t heads, int64_t batches) {
  const bool repeats = (t.stride_s == 0 && rows > 1) || (t.stride_h == 0 && heads > 1) || (t.stride_b == 0 && batches > 1);
  return rows_compatible(t) && !(t.ptr && repeats);
}

}  // namespace fa
