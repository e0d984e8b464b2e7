// The driver's tensor-map encoder, reached through the runtime (the library links no libcuda).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace risa_gb {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled as introduced in CUDA 12.0, or nullptr.
inline EncodeTiled encode_fn() {
   static const EncodeTiled fn = [] {
      void* p = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
              cudaSuccess &&
          q == cudaDriverEntryPointSuccess)
         return reinterpret_cast<EncodeTiled>(p);
      return EncodeTiled(nullptr);
   }();
   return fn;
}

}  // namespace risa_gb
