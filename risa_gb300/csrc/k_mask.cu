// Masking stage: optional min-max normalisation, then the inscribed-circle
// mask (Masking.cu:113-169). The reference normalises with
// thrust::minmax_element + thrust::transform (two passes plus a host read of
// min/max); here a cluster per image writes its min/max to a small
// device workspace and the mask kernel reads them, so nothing syncs with the
// host. Without normalisation the mask is fused into the backprojection.
#include <cooperative_groups.h>

#include <cmath>
#include <cstdint>

#include "kernels.h"

namespace risa_gb {

namespace {
// order-preserving float <-> uint mapping for atomicMin/atomicMax
__device__ __forceinline__ unsigned int f2o(float f) {
   const unsigned int u = __float_as_uint(f);
   return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(unsigned int u) {
   return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Minimum and maximum of one image by a cluster of 8 CTAs: 16-byte loads, four in
// flight, then the CTAs' pairs through distributed shared memory. One launch,
// nothing to initialise (231^2 4.5 us; 8 with 32 CTAs, scalar loads, atomics and an
// initialising launch). Every CTA reaches both cluster barriers.
constexpr int kMinMaxCluster = 8, kMinMaxThreads = 1024;
__global__ void __cluster_dims__(kMinMaxCluster, 1, 1) __launch_bounds__(kMinMaxThreads)
    minmax_cluster(const float* __restrict__ img, int n, unsigned int* __restrict__ mm) {
   namespace cg = cooperative_groups;
   cg::cluster_group cl = cg::this_cluster();
   __shared__ unsigned int s_lo[32], s_hi[32], s_pair[2];
   const int b = blockIdx.y;
   const float* im = img + (size_t)b * n;
   float lo = INFINITY, hi = -INFINITY;
   auto take = [&](float v) {
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
   };
   const int tid = blockIdx.x * kMinMaxThreads + threadIdx.x, nt = kMinMaxCluster * kMinMaxThreads;
   const int n4 = (reinterpret_cast<uintptr_t>(im) & 15) == 0 ? n / 4 : 0;
#pragma unroll 4
   for (int i = tid; i < n4; i += nt) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(im) + i);
      take(v.x);
      take(v.y);
      take(v.z);
      take(v.w);
   }
#pragma unroll 4
   for (int i = 4 * n4 + tid; i < n; i += nt) take(__ldg(im + i));
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const unsigned wlo = __reduce_min_sync(~0u, f2o(lo)), whi = __reduce_max_sync(~0u, f2o(hi));
   if (lane == 0) {
      s_lo[warp] = wlo;
      s_hi[warp] = whi;
   }
   __syncthreads();
   if (warp == 0) {
      const unsigned clo = __reduce_min_sync(~0u, s_lo[lane]), chi = __reduce_max_sync(~0u, s_hi[lane]);
      if (lane == 0) {
         s_pair[0] = clo;
         s_pair[1] = chi;
      }
   }
   cl.sync();
   if (blockIdx.x == 0 && threadIdx.x == 0) {
      unsigned rlo = 0xFFFFFFFFu, rhi = 0u;
      for (int q = 0; q < kMinMaxCluster; ++q) {
         const unsigned* p = cl.map_shared_rank(&s_pair[0], q);
         rlo = min(rlo, p[0]);
         rhi = max(rhi, p[1]);
      }
      mm[2 * b] = rlo;
      mm[2 * b + 1] = rhi;
   }
   cl.sync();  // the other CTAs' shared memory stays alive until the pairs are read
}

__global__ void mask_apply(float* __restrict__ img, int N, float value, int normalize,
                           const unsigned int* __restrict__ mm, int masking, float lim) {
   const int x = blockIdx.x * blockDim.x + threadIdx.x;
   const int y = blockIdx.y;
   const int b = blockIdx.z;
   if (x >= N) return;
   float* p = img + ((size_t)b * N + y) * N + x;
   float v = *p;
   if (normalize) {
      const float mn = o2f(mm[2 * b]), mx = o2f(mm[2 * b + 1]);
      v = (v - mn) / (mx - mn);
   }
   if (masking) {
      const float c = (float)((N - 1.0) * 0.5);
      const float dx = (float)x - c, dy = (float)y - c;
      if (dx * dx + dy * dy > lim) v = value;
   }
   *p = v;
}
}  // namespace

cudaError_t launch_mask(float* img, int batch, int N, float value, int normalize,
                        float* ws_minmax, int masking, cudaStream_t st) {
   if (batch <= 0) return cudaSuccess;
   unsigned int* mm = reinterpret_cast<unsigned int*>(ws_minmax);
   if (normalize) {
      dim3 g(kMinMaxCluster, batch);
      minmax_cluster<<<g, kMinMaxThreads, 0, st>>>(img, N * N, mm);
   }
   // the largest float not above N^2 / 4: a float exceeds one as it exceeds the other
   const double r2 = (double)N * (double)N * 0.25;
   float lim = (float)r2;
   if ((double)lim > r2) lim = std::nextafter(lim, 0.f);
   dim3 grid((N + 127) / 128, N, batch);
   mask_apply<<<grid, 128, 0, st>>>(img, N, value, normalize, mm, masking, lim);
   return cudaGetLastError();
}

}  // namespace risa_gb
