// Host-side construction of TMA descriptors.  The one driver entry point needed, ``cuTensorMapEncodeTiled``, is
// resolved at run time so that the library links against the CUDA runtime only.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace b2 {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A host thread that has made no CUDA runtime call yet has no current context (PyTorch's autograd worker thread on
// device 0 is one: it never needs to switch devices), and the driver entry point then answers
// CUDA_ERROR_INVALID_CONTEXT (201).  ``cudaFree(nullptr)`` binds the primary context of the current device; once per
// thread.
static inline void bind_primary_context() {
  static thread_local bool bound = false;
  if (!bound) {
    cudaFree(nullptr);
    bound = true;
  }
}

static inline EncodeTiledFn encode_fn() {
  bind_primary_context();
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &res) == cudaSuccess &&
        res == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// 2-D bf16 tensor [outer, inner] with row pitch ``pitch_elems``; box = [box_outer, 64] elements, 128B swizzle.
static inline int make_map(CUtensorMap* map, const void* base, long long inner, long long outer, long long pitch_elems,
                    int box_outer) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch_elems) * 2};
  cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_outer)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// fp32 result [experts, rows, cols] with row pitch ``pitch_elems`` and expert pitch ``expert_elems``, as the epilogue's
// stores address it: boxes of 32 rows x 32 columns, 128B swizzle.
static inline int make_out_map(CUtensorMap* map, const void* base, long long cols, long long rows, long long experts,
                               long long pitch_elems, long long expert_elems) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(experts)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(pitch_elems) * 4, static_cast<cuuint64_t>(expert_elems) * 4};
  cuuint32_t box[3] = {32, 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

}  // namespace b2
