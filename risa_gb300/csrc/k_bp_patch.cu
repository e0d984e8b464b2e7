// Linear pixel-driven backprojection of slice batches, 2 x 2 pixel patches per
// thread (the batch form of backProjectLinear, Backprojection.cu:238-271).
//
// What bounds a linear backprojection is the shared-memory data path: a
// (midpoint, difference) record per pixel, angle and slice is 8 B of every
// 128 B/clk (bp_linear_async, k_bp.cu: 23.8 ms per 512 slices of 1024 x 1024
// -> 512^2, 0.90 of that bound). Here a thread owns a 2 x 2 pixel patch of 4, 8
// or 16 slices and reads each detector bin its patch touches once: with
// A = |a|, B = |b| (bins per pixel along x and y) the patch spans A + B bins,
// so floor(A + B) + 3 bins serve 4 pixels -- 5 loads of 16 B at 2 bins per
// pixel and 4 at 1, where the records took 8. The form for large batches leaves the last
// out where its weight is 0: 4.55 B per update and slice at 2 bins per pixel, 15.7 ms
// for the launch above, 0.78 of the measured 40 TB/s counting the pixels in the circle alone.
//
//   * A pixel at offset o from the patch's lowest coordinate k + g (g in [0, 1])
//     reads the three bins m .. m + 2 around g + o, m = floor(o), with the hat
//     weights of linear interpolation max(0, 1 - |g + o - m - 1 -+ 1|) and
//     1 - |g + o - m - 1|; one of the outer two is 0. m is the same for every
//     thread of an angle, so the bins are registers with compile-time indices:
//     the angles are sorted by (sign of a, sign of b, m of the three offset
//     pixels) and every chunk of angles runs the loop instantiated for its class.
//     A negative a or b mirrors the patch: the accumulators are exchanged once,
//     where the sign changes.
//   * The rows are staged as they are, four slices to a 16-byte entry
//     ([slice quad][angle][bin][4]): no (mid, diff) pairs, so half the bytes in
//     global memory and in the staging copies, and no padding: bins outside the
//     detector are the zeros a tensor-map copy fills in.
//   * A warp is QL slice quads x 32 / QL patches. With QL = 8 the 8 lanes of a
//     128-bit load phase read one bin of 8 quads, whose rows lie an odd number
//     of entries apart: conflict-free whatever the bins per pixel.
//
// One warp of the CTA forms the windows and fills NST shared-memory stages of
// ACH angles with cp.async.bulk.tensor (one box per angle: the tile's bins of
// all the CTA's quads), each completing on its stage's `full` mbarrier; the other
// warps release a stage on its `empty` mbarrier. With the refill done by one of
// the working warps, as in bp_linear_async, the same loop took 18.0 ms instead
// of 15.8 (512 slices of 1024 x 1024 -> 512^2). Waits are bounded; on timeout the
// CTA records the error and leaves without output.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "async_copy.h"
#include "f32x2.cuh"
#include "kernels.h"
#include "patch_window.cuh"
#include "risa_gb300.h"
#include "tensor_map.h"

namespace risa_gb {

namespace {
constexpr int kTile = 16;  // pixels per tile side
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kMagicBits = 0x4B400000;

struct PatchArgs {
   const BPPatchAngle* ang;  // [Pp] in plan order
   const int* nonfinite;     // per slice quad: its slices that hold an infinity or a NaN; or nullptr
   const float4* quads;      // [quad][angle][bin] (the rows the tensor map covers)
   float* img;
   int* err;
   int N, Pp, Dp, batch, n_quads, wlen;
   float norm, mask_value;
   int masking;
};
struct PatchSegs {
   uint32_t seg[kPatchMaxSegs];
   int n_segs;
};
struct PatchPlanParam : PatchSegs {
   float A[kPatchAngles], B[kPatchAngles];
};

typedef unsigned long long u64;

__device__ __forceinline__ ulonglong2 lds_quad(uint32_t addr) {
   ulonglong2 v;
   asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr));
   return v;
}

// The same load for the lanes with r > 0, zeros elsewhere: a load phase whose
// lanes all skip it costs no wavefront.
__device__ __forceinline__ ulonglong2 lds_quad_if(uint32_t addr, float r) {
   ulonglong2 v;
   asm volatile(
       "{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %3, 0f00000000;\n\tmov.u64 %0, 0;\n\tmov.u64 %1, 0;\n\t"
       "@p ld.shared.v2.u64 {%0, %1}, [%2];\n\t}"
       : "=&l"(v.x), "=&l"(v.y)
       : "r"(addr), "f"(r));
   return v;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
   asm volatile(
       "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
           "r"(async::smem_u32(dst)),
       "l"(map), "r"(async::smem_u32(bar)), "r"(x), "r"(y), "r"(z)
       : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
   asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(async::smem_u32(bar)) : "memory");
}

// One angle of one patch: addr is the shared address of bin k of this thread's
// first quad, f = g - 1/2.
template <int MA, int MB, int MAB, int SQ, bool PRED>
__device__ __forceinline__ void patch_angle(uint32_t addr, uint32_t qstep, float f, float A, float B,
                                            u64 (&acc)[SQ][2][4]) {
   constexpr int m[4] = {0, MA, MB, MAB};
   // coordinate of each pixel relative to its middle bin m + 1, in [-1, 1]
   const float r1 = (f + A) - (MA + 0.5f), r2 = (f + B) - (MB + 0.5f), r3 = (f + (A + B)) - (MAB + 0.5f);
   const float r[4] = {0.f, r1, r2, r3};
   float w[4][3];
   w[0][0] = 0.5f - f;  // the lowest pixel lies between bins 0 and 1
   w[0][1] = 0.5f + f;
   w[0][2] = 0.f;
#pragma unroll
   for (int p = 1; p < 4; ++p) {
      w[p][0] = __saturatef(-r[p]);
      w[p][1] = 1.f - fabsf(r[p]);
      w[p][2] = __saturatef(r[p]);
   }
#pragma unroll
   for (int e = 0; e < MAB + 3; ++e) {
      ulonglong2 q[SQ];
#pragma unroll
      for (int s = 0; s < SQ; ++s) {
         const uint32_t at = addr + (uint32_t)s * qstep + (uint32_t)e * 16u;
         q[s] = PRED && e == MAB + 2 ? lds_quad_if(at, r3) : lds_quad(at);
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) {
         const int d = e - m[p];
         if (d < 0 || d > (p == 0 ? 1 : 2)) continue;
         const u64 w2 = f2_pack(w[p][d], w[p][d]);
#pragma unroll
         for (int s = 0; s < SQ; ++s) {
            acc[s][0][p] = f2_fma(w2, q[s].x, acc[s][0][p]);
            acc[s][1][p] = f2_fma(w2, q[s].y, acc[s][1][p]);
         }
      }
   }
}

template <int SQ>
__device__ __forceinline__ void flip(u64 (&acc)[SQ][2][4], bool x, bool y) {
#pragma unroll
   for (int s = 0; s < SQ; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
         u64* v = acc[s][h];
         u64 t;
         if (x) t = v[0], v[0] = v[1], v[1] = t, t = v[2], v[2] = v[3], v[3] = t;
         if (y) t = v[0], v[0] = v[2], v[2] = t, t = v[1], v[1] = v[3], v[3] = t;
      }
}

// The slices of a CTA's tile whose rows hold an infinity or a NaN (bit j of the
// quad's flag: slice j), by the general two-bin rule: the patches also multiply a
// third bin by a zero weight, which would carry it one pixel further. The CTA's
// other slices have their pixels from the patches. A flagged slice at a time, one to
// three pixels per thread, the windows of C angles in the copies' stages (16 rows of
// 16-byte entries for every quad); all threads of the CTA, before the first copy (after
// the last patch the call alone cost the finite CTAs 0.8%). 64 slices of 512^2 x 1024
// angles 2.2 ms, with one bad sample 3.3; 108 with every quad of the CTA by scalar loads and
// FP64 coordinates, 3.5 with the flagged quad's four slices at once.
template <int Q, int NT>
__device__ __noinline__ void patch_general_tile(const PatchArgs& g) {
   constexpr int C = Q == 1 ? 40 : 64, PX = (kTile * kTile + NT - 1) / NT;  // angles per chunk, pixels per thread
   extern __shared__ __align__(128) unsigned char smem_raw[];
   const int N = g.N, Dp = g.Dp, wlen = g.wlen, x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   float4* tab = reinterpret_cast<float4*>(smem_raw);  // a, b, window-relative coordinate, first bin
   float* win = reinterpret_cast<float*>(tab + C);     // [C][wlen]
   for (int sl = 4 * blockIdx.z * Q; sl < min(4 * (int)(blockIdx.z + 1) * Q, g.batch); ++sl) {
      if (!(__ldg(g.nonfinite + (sl >> 2)) >> (sl & 3) & 1)) continue;
      float acc[PX];
#pragma unroll
      for (int r = 0; r < PX; ++r) acc[r] = 0.f;
      for (int c0 = 0; c0 < g.Pp; c0 += C) {
         const int na = min(C, g.Pp - c0);
         __syncthreads();
         if (threadIdx.x < na) {
            const BPPatchAngle t = g.ang[c0 + threadIdx.x];
            int w0;
            float rel;
            patch_window<1>(t, x0 + (t.a_hi < 0.f ? kTile - 1 : 0), y0 + (t.b_hi < 0.f ? kTile - 1 : 0), &w0, &rel);
            tab[threadIdx.x] = make_float4(t.a_hi, t.b_hi, rel, __int_as_float(w0));
         }
         __syncthreads();
         for (int ai = warp; ai < na; ai += NT / 32) {
            const float* row = reinterpret_cast<const float*>(
                                   g.quads + ((size_t)(sl >> 2) * g.Pp + __ldg(&g.ang[c0 + ai].index)) * Dp) + (sl & 3);
            const int w0 = __float_as_int(tab[ai].w);
            for (int m = lane; m < wlen; m += 32)
               win[ai * wlen + m] = (unsigned)(w0 + m) < (unsigned)Dp ? __ldg(row + 4 * (w0 + m)) : 0.f;
         }
         __syncthreads();
#pragma unroll 2
         for (int ai = 0; ai < na; ++ai) {
            const float4 e = tab[ai];
#pragma unroll
            for (int r = 0; r < PX; ++r) {
               const int p = (int)threadIdx.x + r * NT, px = p % kTile, py = p / kTile;
               if (p >= kTile * kTile) break;
               const float fx = (float)(e.x < 0.f ? kTile - 1 - px : px), fy = (float)(e.y < 0.f ? kTile - 1 - py : py);
               const float t = fmaf(fy, fabsf(e.y), fmaf(fx, fabsf(e.x), e.z));
               const float fl = floorf(t), f = (t - fl) - 0.5f;
               const float* w = win + ai * wlen + min((int)fl, wlen - 2);  // the patches of this tile reach as many bins
               const float u = w[0], v = w[1];
               acc[r] = fmaf(f, v - u, acc[r] + 0.5f * (u + v));
            }
         }
      }
      const float c = 0.5f * (float)(N - 1), lim = (float)N * (float)N * 0.25f;
#pragma unroll
      for (int r = 0; r < PX; ++r) {
         const int p = (int)threadIdx.x + r * NT, x = x0 + p % kTile, y = y0 + p / kTile;
         if (p >= kTile * kTile || x >= N || y >= N) continue;
         const float dx = (float)x - c, dy = (float)y - c;
         const bool out = g.masking && dx * dx + dy * dy > lim;
         g.img[((size_t)sl * N + y) * N + x] = out ? g.mask_value : acc[r] * g.norm;
      }
   }
}

template <int SQ, int QL, int ACH, int NST, int MINB, bool PRED>
__global__ void __launch_bounds__(64 * QL + 32, MINB)
    bp_patch(const __grid_constant__ CUtensorMap map, const __grid_constant__ PatchArgs g, const __grid_constant__ PatchPlanParam pp) {
   constexpr int NW = 2 * QL, Q = QL * SQ;  // consumer warps, slice quads of the CTA
   extern __shared__ __align__(128) unsigned char smem_raw[];
   __shared__ uint64_t full[NST], empty[NST];
   __shared__ float4 s_rel[NST][ACH / 4];
   __shared__ volatile int s_fail;

   const int N = g.N;
   const int x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile, q0 = blockIdx.z * Q;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   bool flagged = false;
   if (g.nonfinite) {
#pragma unroll 1
      for (int i = q0; i < min(q0 + Q, g.n_quads); ++i) flagged |= __ldg(g.nonfinite + i) != 0;
      if (flagged) {
         patch_general_tile<Q, (NW + 1) * 32>(g);
         asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // its stages are the copies' from the next barrier on
      }
   }
   const float c = 0.5f * (float)(N - 1);
   const float lim = (float)N * (float)N * 0.25f;
   // whether some pixel of the block lies inside the circle (exact, as in bp_linear_async)
   auto inside = [&](int xa, int ya, int w, int h) {
      const float nx = fminf(fmaxf(c, (float)xa), (float)(xa + w - 1)) - c;
      const float ny = fminf(fmaxf(c, (float)ya), (float)(ya + h - 1)) - c;
      return !g.masking || nx * nx + ny * ny <= lim;
   };
   // a consumer warp's pixel block in the tile
   constexpr int BW = QL == 8 ? 4 : QL == 1 ? 16 : 8, BH = 128 / QL / BW;
   auto block_x = [](int w) { return w % (kTile / BW) * BW; };
   auto block_y = [](int w) { return w / (kTile / BW) * BH; };

   const bool tile_live = inside(x0, y0, kTile, kTile);
   const uint32_t pitch = (uint32_t)g.wlen * 16u;     // bytes between the rows of two quads
   const uint32_t angle_bytes = pitch * (uint32_t)Q;  // one angle's box
   if (threadIdx.x == 0) {
      int live_warps = 0;
      for (int w = 0; w < NW; ++w) live_warps += inside(x0 + block_x(w), y0 + block_y(w), BW, BH);
      for (int i = 0; i < NST; ++i) {
         async::mbar_init(&full[i], 1);
         async::mbar_init(&empty[i], max(live_warps, 1));
      }
      s_fail = 0;
      async::mbar_init_fence();
   }
   __syncthreads();

   if (warp == NW) {
      // ---- producer: windows and copies of every chunk
      int st = 0;
      uint32_t round = 0;
      for (int si = 0; tile_live && si < pp.n_segs && !s_fail; ++si) {
         const uint32_t d = pp.seg[si];
         const int pos = (int)(d & 0xFFFu), n = (int)((d >> 12) & 0xFFFu);
         const int cx = x0 + ((d >> 28) & 1u ? kTile - 1 : 0), cy = y0 + ((d >> 29) & 1u ? kTile - 1 : 0);
         for (int a0 = 0; a0 < n; a0 += ACH) {
            const int na = min(ACH, n - a0);
            float rel = 0.f;
            int w0 = 0, ang = 0;
            if (lane < na) {
               const BPPatchAngle t = g.ang[pos + a0 + lane];
               patch_window<1>(t, cx, cy, &w0, &rel);
               ang = t.index;
            }
            if (round > 0 && !__all_sync(~0u, async::mbar_wait(&empty[st], (round - 1) & 1u, g.err, 5))) {
               s_fail = 1;
               break;
            }
            if (lane < ACH) reinterpret_cast<float*>(&s_rel[st][0])[lane] = rel - 0.5f;
            __syncwarp();
            if (lane == 0) async::mbar_arrive_expect_tx(&full[st], (uint32_t)na * angle_bytes);
            __syncwarp();
            if (lane < na)
               tma_load_3d(smem_raw + (size_t)(st * ACH + lane) * angle_bytes, &map, &full[st], 4 * w0, ang, q0);
            if (++st == NST) st = 0, ++round;
         }
      }
      // the copies still in flight land before the CTA ends
      for (int i = 0; i < NST; ++i) {
         const uint32_t issued = round + (i < st ? 1u : 0u);
         if (issued > 0) async::mbar_wait_quiet(&full[i], (issued - 1) & 1u);
      }
      __syncthreads();
      return;
   }

   // ---- consumers
   const int ql = lane % QL, pl = lane / QL;
   // this thread's patch in the warp's block: the patches of a load phase are neighbours
   int px, py;
   if (QL == 8) px = pl & 1, py = pl >> 1;
   else if (QL == 4) px = pl & 3, py = pl >> 2;
   else if (QL == 2) px = (pl & 1) + ((pl >> 1) & 2), py = ((pl >> 1) & 1) + ((pl >> 2) & 2);
   else px = (pl & 3) + ((pl >> 1) & 4), py = ((pl >> 2) & 1) + ((pl >> 3) & 2);
   const int xp = block_x(warp) + 2 * px, yp = block_y(warp) + 2 * py;  // patch origin in the tile

   u64 acc[SQ][2][4];
#pragma unroll
   for (int s = 0; s < SQ; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
         for (int p = 0; p < 4; ++p) acc[s][h][p] = 0ull;

   const uint32_t sbase = async::smem_u32(smem_raw) + (uint32_t)ql * pitch - ((uint32_t)kMagicBits << 4);
   if (tile_live && inside(x0 + block_x(warp), y0 + block_y(warp), BW, BH)) {
      uint32_t signs = 0;  // bit 0: x mirrored, bit 1: y mirrored
      int st = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int si = 0; si < pp.n_segs && ok; ++si) {
         const uint32_t d = pp.seg[si];
         const int pos = (int)(d & 0xFFFu), n = (int)((d >> 12) & 0xFFFu);
         const uint32_t sg = d >> 28;
         if (sg != signs) {
            flip<SQ>(acc, (sg ^ signs) & 1u, ((sg ^ signs) >> 1) & 1u);
            signs = sg;
         }
         const float fx = (float)((sg & 1u) ? kTile - 2 - xp : xp), fy = (float)((sg & 2u) ? kTile - 2 - yp : yp);
         auto run = [&](auto cls) {
            constexpr int CL = decltype(cls)::value;
#pragma unroll 1
            for (int a0 = 0; a0 < n; a0 += ACH) {
               if (!async::mbar_wait(&full[st], phase, g.err, 5)) {
                  ok = false;
                  break;
               }
               const uint32_t stage = sbase + (uint32_t)(st * ACH) * angle_bytes;
               auto angle = [&](int ai, float rel) {
                  const float A = pp.A[pos + a0 + ai], B = pp.B[pos + a0 + ai];
                  const float tm = fmaf(fy, B, fmaf(fx, A, rel));
                  const float v = tm + kMagic;
                  const float f = tm - (v - kMagic);
                  const uint32_t addr = stage + (uint32_t)ai * angle_bytes + ((uint32_t)__float_as_int(v) << 4);
                  patch_angle<(CL >> 3), (CL >> 2) & 1, CL & 3, SQ, PRED>(addr, pitch * QL, f, A, B, acc);
               };
               if (n - a0 >= ACH) {
#pragma unroll 1
                  for (int a4 = 0; a4 < ACH; a4 += 4) {
                     const float4 r4 = s_rel[st][a4 >> 2];
                     angle(a4, r4.x);
                     angle(a4 + 1, r4.y);
                     angle(a4 + 2, r4.z);
                     angle(a4 + 3, r4.w);
                  }
               } else {
#pragma unroll 1
                  for (int ai = 0; ai < n - a0; ++ai) angle(ai, reinterpret_cast<const float*>(&s_rel[st][0])[ai]);
               }
               __syncwarp();
               if (lane == 0) mbar_arrive(&empty[st]);
               if (++st == NST) st = 0, phase ^= 1u;
            }
         };
         switch ((d >> 24) & 15u) {  // class: MA << 3 | MB << 2 | MAB
            case 0: run(std::integral_constant<int, 0>{}); break;
            case 1: run(std::integral_constant<int, 1>{}); break;
            case 5: run(std::integral_constant<int, 5>{}); break;
            case 6: run(std::integral_constant<int, 6>{}); break;
            case 9: run(std::integral_constant<int, 9>{}); break;
            case 10: run(std::integral_constant<int, 10>{}); break;
            default: run(std::integral_constant<int, 14>{}); break;
         }
      }
      if (!ok) s_fail = 1;
      flip<SQ>(acc, signs & 1u, (signs >> 1) & 1u);
   }
   __syncthreads();
   if (s_fail) return;  // a wait gave up (recorded in g.err): no output
   auto store = [&](auto skip) {  // skip: but the flagged slices, which are written already
#pragma unroll
      for (int s = 0; s < SQ; ++s)
#pragma unroll
         for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int p = 0; p < 4; ++p) {
               float v[2];
               f2_unpack(acc[s][h][p], v[0], v[1]);
               const int x = x0 + xp + (p & 1), y = y0 + yp + (p >> 1);
               if (x >= N || y >= N) continue;
               bool out = false;
               if (g.masking) {
                  const float dx = (float)x - c, dy = (float)y - c;
                  out = dx * dx + dy * dy > lim;
               }
#pragma unroll
               for (int j = 0; j < 2; ++j) {
                  const int sl = 4 * (q0 + s * QL + ql) + 2 * h + j;
                  if (sl >= g.batch) continue;
                  if (decltype(skip)::value && (__ldg(g.nonfinite + (sl >> 2)) >> (sl & 3) & 1)) continue;
                  g.img[((size_t)sl * N + y) * N + x] = out ? g.mask_value : v[j] * g.norm;
               }
            }
   };
   if (flagged) store(std::true_type());
   else store(std::false_type());
}

// ---- one or two slices: the same patches over the sinogram itself ------------
// A frame at a time there are no slices to share a pixel's weights and a 16 x 16
// tile is 64 patches, too few warps to hide the shared-memory latency. Here the
// G groups of a CTA take the angles of a chunk in turn over the same patches and
// add their sums in group order at the end, the rows come straight from the
// sinogram (no staging pass; windows start at a multiple of 4 bins, as the copy
// needs), and a pixel reads its two bins by selecting the outer one, so
// infinities and NaN stay where the general kernel leaves them.
// A stage is refilled by all working warps: with one producer warp as
// in bp_patch the same loop took 141 us, with 16-byte cp.async pieces instead of a
// box per angle 134. One slice of 1024 x 1024 -> 512^2: 119 us, 91 with symmetric
// sets (quads 263, pairs_s1_a32 229); 512 x 256 -> 256^2: 28 and 27 us (66, 80).
// Bound by issue (70%), half of it on the integer and select pipe.
template <int R>
constexpr int kRowsACH = 64 / R;  // angles per chunk, R rows each

struct RowsArgs {
   const BPPatchAngle* ang;
   const float* sino;
   float* img;   // SYM: the partial images [4][S][N][N]
   int* err;
   int N, Pp, Dp, wlen;
   float norm, mask_value;
   int masking;
};

__device__ __forceinline__ float lds_f32(uint32_t addr) {
   float v;
   asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
   return v;
}

// off: the offset pixels' coordinates relative to their middle bins at f = 0.
template <int MA, int MB, int MAB, int R>
__device__ __forceinline__ void rows_angle(uint32_t addr, uint32_t sstep, float f, float4 off, float (&acc)[R][4]) {
   constexpr int m[4] = {0, MA, MB, MAB};
   const float r[4] = {0.f, f + off.x, f + off.y, f + off.z};
#pragma unroll
   for (int s = 0; s < R; ++s) {
      float q[MAB + 3];
#pragma unroll
      for (int e = 0; e < MAB + 3; ++e) q[e] = lds_f32(addr + (uint32_t)s * sstep + (uint32_t)e * 4u);
      acc[s][0] = fmaf(0.5f - f, q[0], acc[s][0]);
      acc[s][0] = fmaf(0.5f + f, q[1], acc[s][0]);
#pragma unroll
      for (int p = 1; p < 4; ++p) {
         const float outer = r[p] < 0.f ? q[m[p]] : q[m[p] + 2];
         acc[s][p] = fmaf(1.f - fabsf(r[p]), q[m[p] + 1], acc[s][p]);
         acc[s][p] = fmaf(fabsf(r[p]), outer, acc[s][p]);
      }
   }
}

// SYM: the rows of four angles at once. With the angles i pi / Pp of an unrotated
// scan, theta, pi - theta, pi/2 + theta and pi/2 - theta (rows i, Pp - i, Pp/2 + i,
// Pp/2 - i) see a pixel, its x mirror, its quarter turn and its transpose at the
// same ray coordinate, so the bin index and the weights of a patch serve four
// rows, as they serve the slices of a quad in bp_patch. The sums go to four
// partial images (pixel = where that row's contribution belongs), which
// bp_patch_combine adds with the angles that are not in a set of four (0, Pp/2 and,
// where Pp is a multiple of 4, Pp/4 and 3 Pp/4).
template <int S, int G, bool SYM>
__global__ void __launch_bounds__(64 * G)
    bp_patch_rows(const __grid_constant__ CUtensorMap map, const __grid_constant__ RowsArgs g,
                  const __grid_constant__ PatchSegs pp) {
   constexpr int R = SYM ? 4 * S : S, ACH = kRowsACH<R>;  // rows per angle, angles per chunk
   extern __shared__ __align__(128) unsigned char smem_raw[];
   __shared__ uint64_t full[2], empty[2];
   // per angle: (|a|, |b|, window-relative coordinate - 1/2), then rows_angle's offsets
   __shared__ float4 s_par[2][ACH][2];
   __shared__ volatile int s_fail;

   const int N = g.N;
   const int x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const float c = 0.5f * (float)(N - 1);
   const float lim = (float)N * (float)N * 0.25f;
   auto inside = [&](int xa, int ya, int w, int h) {
      const float nx = fminf(fmaxf(c, (float)xa), (float)(xa + w - 1)) - c;
      const float ny = fminf(fmaxf(c, (float)ya), (float)(ya + h - 1)) - c;
      return !g.masking || nx * nx + ny * ny <= lim;
   };
   // a group's two warps cover 16 x 8 pixels each; halves outside the circle are left out
   const bool live0 = inside(x0, y0, kTile, kTile / 2), live1 = inside(x0, y0 + kTile / 2, kTile, kTile / 2);
   const int halves = (int)live0 + (int)live1, L = G * halves;  // working warps
   const uint32_t row_bytes = (uint32_t)g.wlen * 4u, angle_bytes = row_bytes * R;
   if (threadIdx.x == 0) {
      for (int i = 0; i < 2; ++i) {
         async::mbar_init(&full[i], max(L, 1));
         async::mbar_init(&empty[i], max(L, 1));
      }
      s_fail = 0;
      async::mbar_init_fence();
   }
   __syncthreads();

   float acc[R][4];
#pragma unroll
   for (int s = 0; s < R; ++s)
#pragma unroll
      for (int p = 0; p < 4; ++p) acc[s][p] = 0.f;
   const int group = warp >> 1;
   const int xp = 2 * ((lane & 3) + ((lane >> 1) & 4));
   const int yp = (warp & 1) * 8 + 2 * (((lane >> 2) & 1) + ((lane >> 3) & 2));

   if ((warp & 1) ? live1 : live0) {
      const int rank = halves == 2 ? warp : group;
      // Refill of a stage with one chunk (angles a0 .. a0 + ACH - 1 of run `d`):
      // every working warp forms the windows of its angles (rank + j L, one per
      // lane) and issues their copies.
      auto refill = [&](uint32_t d, int a0, int st) {
         const int pos = (int)(d & 0xFFFu), na = min(ACH, (int)((d >> 12) & 0xFFFu) - a0);
         const int mine = na > rank ? (na - rank + L - 1) / L : 0;
         int w0 = 0, row = 0;
         if (lane < mine) {
            const int a = rank + lane * L;
            const BPPatchAngle t = g.ang[pos + a0 + a];
            float rel;
            patch_window<4>(t, x0 + ((d >> 28) & 1u ? kTile - 1 : 0), y0 + ((d >> 29) & 1u ? kTile - 1 : 0), &w0, &rel);
            row = t.index;
            const float A = fabsf(t.a_hi), B = fabsf(t.b_hi);
            const uint32_t cls = (d >> 24) & 15u;
            s_par[st][a][0] = make_float4(A, B, rel - 0.5f, 0.f);
            s_par[st][a][1] = make_float4(A - ((float)(cls >> 3) + 0.5f), B - ((float)((cls >> 2) & 1u) + 0.5f),
                                          (A + B) - ((float)(cls & 3u) + 0.5f), 0.f);
         }
         __syncwarp();
         if (lane == 0) async::mbar_arrive_expect_tx(&full[st], (uint32_t)mine * angle_bytes);
         __syncwarp();
         if (lane < mine) {
            unsigned char* dst = smem_raw + (size_t)(st * ACH + rank + lane * L) * angle_bytes;
            tma_load_3d(dst, &map, &full[st], w0, row, 0);
            if (SYM) {
               const uint32_t step = row_bytes * S;
               tma_load_3d(dst + step, &map, &full[st], w0, g.Pp - row, 0);
               tma_load_3d(dst + 2 * step, &map, &full[st], w0, g.Pp / 2 + row, 0);
               tma_load_3d(dst + 3 * step, &map, &full[st], w0, g.Pp / 2 - row, 0);
            }
         }
      };
      const uint32_t sbase = async::smem_u32(smem_raw) - ((uint32_t)kMagicBits << 2);
      uint32_t signs = 0;
      auto flip1 = [&](uint32_t f) {
#pragma unroll
         for (int s = 0; s < R; ++s) {
            float* v = acc[s];
            float t;
            if (f & 1u) t = v[0], v[0] = v[1], v[1] = t, t = v[2], v[2] = v[3], v[3] = t;
            if (f & 2u) t = v[0], v[0] = v[2], v[2] = t, t = v[1], v[1] = v[3], v[3] = t;
         }
      };
      refill(pp.seg[0], 0, 0);
      int ch = 0;  // chunks done
      bool ok = true;
      for (int si = 0; si < pp.n_segs && ok; ++si) {
         const uint32_t d = pp.seg[si];
         const int n = (int)((d >> 12) & 0xFFFu);
         const uint32_t sg = (d >> 28) & 3u;
         flip1(sg ^ signs);
         signs = sg;
         const float fx = (float)((sg & 1u) ? kTile - 2 - xp : xp), fy = (float)((sg & 2u) ? kTile - 2 - yp : yp);
         auto run = [&](auto cls) {
            constexpr int CL = decltype(cls)::value;
#pragma unroll 1
            for (int a0 = 0; a0 < n; a0 += ACH, ++ch) {
               const int st = ch & 1;
               // the next chunk into the other stage, once every warp has left it
               const bool more = a0 + ACH < n;
               if (more || si + 1 < pp.n_segs) {
                  if (ch > 0 && !async::mbar_wait(&empty[st ^ 1], (uint32_t)((ch - 1) >> 1) & 1u, g.err, 5)) {
                     ok = false;
                     break;
                  }
                  refill(more ? d : pp.seg[si + 1], more ? a0 + ACH : 0, st ^ 1);
               }
               if (!async::mbar_wait(&full[st], (uint32_t)(ch >> 1) & 1u, g.err, 5)) {
                  ok = false;
                  break;
               }
               const uint32_t stage = sbase + (uint32_t)(st * ACH) * angle_bytes;
               auto angle = [&](int ai) {
                  const float4 q = s_par[st][ai][0], off = s_par[st][ai][1];
                  const float tm = fmaf(fy, q.y, fmaf(fx, q.x, q.z));
                  const float v = tm + kMagic;
                  const float f = tm - (v - kMagic);
                  const uint32_t addr = stage + (uint32_t)ai * angle_bytes + ((uint32_t)__float_as_int(v) << 2);
                  rows_angle<(CL >> 3), (CL >> 2) & 1, CL & 3, R>(addr, row_bytes, f, off, acc);
               };
               const int na = min(ACH, n - a0);
               int ai = group;
#pragma unroll 1
               for (; ai + 3 * G < na; ai += 4 * G) {
                  angle(ai);
                  angle(ai + G);
                  angle(ai + 2 * G);
                  angle(ai + 3 * G);
               }
#pragma unroll 1
               for (; ai < na; ai += G) angle(ai);
               __syncwarp();
               if (lane == 0) mbar_arrive(&empty[st]);
            }
         };
         switch ((d >> 24) & 15u) {  // as in bp_patch
            case 0: run(std::integral_constant<int, 0>{}); break;
            case 1: run(std::integral_constant<int, 1>{}); break;
            case 5: run(std::integral_constant<int, 5>{}); break;
            case 6: run(std::integral_constant<int, 6>{}); break;
            case 9: run(std::integral_constant<int, 9>{}); break;
            case 10: run(std::integral_constant<int, 10>{}); break;
            default: run(std::integral_constant<int, 14>{}); break;
         }
      }
      if (!ok) s_fail = 1;
      flip1(signs);
   }
   __syncthreads();  // the stages are no longer read
   if (s_fail) {  // a wait gave up: let the copies in flight land, leave without output
      if (threadIdx.x == 0 && L > 0)
         for (int i = 0; i < 2; ++i)
            for (uint32_t ph = 0; ph < 2; ++ph) async::mbar_wait_quiet(&full[i], ph);
      return;
   }
   float* sums = reinterpret_cast<float*>(smem_raw);  // [group][row][pixel of the tile]
#pragma unroll
   for (int s = 0; s < R; ++s)
#pragma unroll
      for (int p = 0; p < 4; ++p)
         sums[(group * R + s) * kTile * kTile + (yp + (p >> 1)) * kTile + xp + (p & 1)] = acc[s][p];
   __syncthreads();
   for (int i = threadIdx.x; i < R * kTile * kTile; i += 64 * G) {
      const int r = i / (kTile * kTile), e = i % (kTile * kTile);
      // rows 2 and 3 of SYM are transposed: consecutive threads take consecutive y
      const bool turned = SYM && r >= 2 * S;
      const int tx = turned ? e / kTile : e % kTile, ty = turned ? e % kTile : e / kTile;
      const int x = x0 + tx, y = y0 + ty;
      if (x >= N || y >= N) continue;
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < G; ++k) v += sums[(k * R + r) * kTile * kTile + ty * kTile + tx];
      if (SYM) {
         const int j = r / S;
         const int X = j == 0 ? x : j == 1 ? N - 1 - x : j == 2 ? N - 1 - y : y, Y = j < 2 ? y : x;
         g.img[((size_t)r * N + Y) * N + X] = v;
         continue;
      }
      v *= g.norm;
      if (g.masking) {
         const float dx = (float)x - c, dy = (float)y - c;
         if (dx * dx + dy * dy > lim) v = g.mask_value;
      }
      g.img[((size_t)r * N + y) * N + x] = v;
   }
}

// Sum of the four partial images and of the angles outside the symmetric sets
// (given by their coefficients), scaled and masked.
struct CombineArgs {
   const float* part;
   const float* sino;
   float* img;
   BPPatchAngle extra[4];
   int n_extra, N, Pp, Dp;
   float norm, mask_value;
   int masking;
};
template <int S>
__global__ void __launch_bounds__(256) bp_patch_combine(const __grid_constant__ CombineArgs g) {
   const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
   const int N = g.N;
   if (x >= N || y >= N) return;
   const size_t at = (size_t)y * N + x, plane = (size_t)N * N;
   const float c = 0.5f * (float)(N - 1), dx = (float)x - c, dy = (float)y - c;
   const bool out = g.masking && dx * dx + dy * dy > (float)N * (float)N * 0.25f;
   float v[S];
#pragma unroll
   for (int s = 0; s < S; ++s) v[s] = 0.f;
   if (!out) {
#pragma unroll
      for (int s = 0; s < S; ++s) {
         const float* p = g.part + s * plane + at;
         v[s] = (p[0] + p[S * plane]) + (p[2 * S * plane] + p[3 * S * plane]);
      }
      for (int i = 0; i < g.n_extra; ++i) {
         int k;
         float f;
         patch_window<1>(g.extra[i], x, y, &k, &f);
         const bool in0 = (unsigned)k < (unsigned)g.Dp, in1 = (unsigned)(k + 1) < (unsigned)g.Dp;
#pragma unroll
         for (int s = 0; s < S; ++s) {
            const float* row = g.sino + ((size_t)s * g.Pp + g.extra[i].index) * g.Dp + k;
            const float q0 = in0 ? __ldg(row) : 0.f, q1 = in1 ? __ldg(row + 1) : 0.f;
            v[s] = fmaf(f - 0.5f, q1 - q0, v[s] + 0.5f * (q0 + q1));
         }
      }
   }
#pragma unroll
   for (int s = 0; s < S; ++s) g.img[s * plane + at] = out ? g.mask_value : v[s] * g.norm;
}

// Staged rows from a plain sinogram: quads[q][angle][bin] = slices 4q .. 4q + 3
// of the bin, 0 past the batch. Bit j of nonfinite[q] (zero before the launch) is set
// where a row of slice j of the quad holds an infinity or a NaN.
__global__ void __launch_bounds__(256) bp_quads_fill(const float* __restrict__ sino, float4* __restrict__ quads,
                                                     int* __restrict__ nonfinite, int batch, int Pp, int Dp) {
   const int k = blockIdx.x * 256 + threadIdx.x;
   if (k >= Dp) return;
   const int ang = blockIdx.y, q = blockIdx.z;
   float v[4];
#pragma unroll
   for (int j = 0; j < 4; ++j)
      v[j] = 4 * q + j < batch ? __ldg(sino + ((size_t)(4 * q + j) * Pp + ang) * Dp + k) : 0.f;
   quads[((size_t)q * Pp + ang) * Dp + k] = make_float4(v[0], v[1], v[2], v[3]);
   int flags = 0;
#pragma unroll
   for (int j = 0; j < 4; ++j) flags |= isfinite(v[j]) ? 0 : 1 << j;
   if (flags && (flags & ~*reinterpret_cast<volatile int*>(nonfinite + q))) atomicOr(nonfinite + q, flags);
}

// Staged row of one angle and quad, in 16-byte entries: the bins a 16-pixel
// tile reaches, rounded up so that the rows of the QL quads of a load phase
// start in different banks (QL rows 8 / QL entries apart modulo a bank row) and
// an angle's box is a multiple of 128 bytes.
int patch_wlen(float scale, int ql) {
   const int need = (int)std::floor((kTile - 2) * 1.41421357 * (double)scale + 1.01) + 3 +
                    std::min(2, (int)std::floor(1.41421357 * (double)scale));
   const int step = 8 / ql;  // 1, 2, 4, 8
   int w = need;
   if (step == 8) return (need + 7) / 8 * 8;
   while (w % step || (w / step) % 2 == 0) ++w;  // an odd multiple of step
   return w;
}

size_t patch_smem(int sq, int ql, int ach, int nst, int wlen) {
   return (size_t)nst * ach * sq * ql * wlen * 16;
}

template <int SQ, int QL, int MINB, bool PRED = false>
cudaError_t launch_patch(const PatchArgs& args, const PatchPlanParam& pp, float scale, cudaStream_t st) {
   constexpr int ACH = 8, NST = 2;
   PatchArgs a = args;
   a.wlen = patch_wlen(scale, QL);
   const size_t smem = patch_smem(SQ, QL, ACH, NST, a.wlen);
   if (4 * a.wlen > 256 || smem > 220 * 1024) return cudaErrorInvalidConfiguration;
   EncodeTiled enc = encode_fn();
   if (!enc) return cudaErrorNotSupported;
   CUtensorMap map;
   const cuuint64_t dims[3] = {(cuuint64_t)a.Dp * 4, (cuuint64_t)a.Pp, (cuuint64_t)a.n_quads};
   const cuuint64_t strides[2] = {(cuuint64_t)a.Dp * 16, (cuuint64_t)a.Pp * a.Dp * 16};
   const cuuint32_t box[3] = {(cuuint32_t)a.wlen * 4, 1, (cuuint32_t)(SQ * QL)};
   const cuuint32_t estr[3] = {1, 1, 1};
   if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float4*>(a.quads), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
   auto kern = bp_patch<SQ, QL, ACH, NST, MINB, PRED>;
   if (smem > 47 * 1024) {  // with the kernel's static shared memory
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
   }
   const int t = (a.N + kTile - 1) / kTile;
   kern<<<dim3(t, t, (a.n_quads + SQ * QL - 1) / (SQ * QL)), 64 * QL + 32, smem, st>>>(map, a, pp);
   return cudaGetLastError();
}

template <int S, int G, bool SYM>
cudaError_t launch_rows(const RowsArgs& args, const PatchSegs& pp, const BPCfg& cfg,
                        cudaStream_t st) {
   RowsArgs a = args;
   const int need = (int)std::floor((kTile - 2) * 1.41421357 * (double)cfg.scale + 4.01) + 3 +
                    std::min(2, (int)std::floor(1.41421357 * (double)cfg.scale));
   a.wlen = need <= 32 ? 32 : 64;
   constexpr int R = SYM ? 4 * S : S;
   const size_t smem = std::max((size_t)2 * kRowsACH<R> * R * a.wlen * 4, (size_t)G * R * kTile * kTile * 4);
   if (need > 64 || smem > 220 * 1024) return cudaErrorInvalidConfiguration;
   EncodeTiled enc = encode_fn();
   if (!enc) return cudaErrorNotSupported;
   CUtensorMap map;
   const cuuint64_t dims[3] = {(cuuint64_t)a.Dp, (cuuint64_t)a.Pp, (cuuint64_t)S};
   const cuuint64_t strides[2] = {(cuuint64_t)a.Dp * 4, (cuuint64_t)a.Pp * a.Dp * 4};
   const cuuint32_t box[3] = {(cuuint32_t)a.wlen, 1, (cuuint32_t)S};
   const cuuint32_t estr[3] = {1, 1, 1};
   if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(a.sino), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
   auto kern = bp_patch_rows<S, G, SYM>;
   if (smem > 47 * 1024) {  // with the kernel's static shared memory
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
   }
   const int t = (a.N + kTile - 1) / kTile;
   kern<<<dim3(t, t), 64 * G, smem, st>>>(map, a, pp);
   return cudaGetLastError();
}
}  // namespace

namespace {
void split(double v, float* hi, float* lo) {
   *hi = (float)v;
   *lo = (float)(v - (double)*hi);
}
// Class and signs of an angle: MA << 3 | MB << 2 | MAB, then (a < 0) | (b < 0) << 1
// in bits 4 and 5; -1 outside the kernel's range.
int patch_group(float a, float b) {
   const float A = std::fabs(a), B = std::fabs(b);
   if (!(A <= 2.f && B <= 2.f && A + B < 3.f)) return -1;
   const int ma = A >= 1.f, mb = B >= 1.f;
   // the offset lies in [m, m + 1]; at an integer either end serves
   const int mab = std::min({(int)(A + B), 2, ma + mb + 1});
   if (A + B - (float)mab > 1.f) return -1;
   return ((a < 0.f ? 1 : 0) | (b < 0.f ? 2 : 0)) << 4 | ma << 3 | mb << 2 | mab;
}
BPPatchAngle patch_angle_of(const double* ad, const double* bd, const double* t0, int i) {
   BPPatchAngle t;
   split(t0[i], &t.t0_hi, &t.t0_lo);
   split(ad[i], &t.a_hi, &t.a_lo);
   split(bd[i], &t.b_hi, &t.b_lo);
   t.index = i;
   t.pad = 0;
   return t;
}
// Runs of equal groups: first | n << 12 | class << 24 | signs << 28.
std::vector<uint32_t> patch_runs(const std::vector<int>& groups) {
   std::vector<uint32_t> segs;
   for (size_t i = 0; i < groups.size();) {
      size_t n = 1;
      while (i + n < groups.size() && groups[i + n] == groups[i]) ++n;
      segs.push_back((uint32_t)i | (uint32_t)n << 12 | (uint32_t)(groups[i] & 15) << 24 |
                     (uint32_t)(groups[i] >> 4) << 28);
      i += n;
   }
   return segs;
}
}  // namespace

bool bp_patch_plan(const float* a, const float* b, const double* ad, const double* bd, const double* t0, int Pp,
                   float scale, bool unrotated, BPPatchPlan* plan) {
   *plan = BPPatchPlan();
   if (Pp < 1 || Pp > kPatchAngles || !(scale > 0.f) || scale > 2.f) return false;
   std::vector<std::pair<int, int>> keys(Pp);  // (group, angle)
   for (int i = 0; i < Pp; ++i) {
      keys[i] = {patch_group(a[i], b[i]), i};
      if (keys[i].first < 0 || !std::isfinite(t0[i])) return false;
   }
   std::sort(keys.begin(), keys.end());
   std::vector<int> groups;
   for (const auto& k : keys) {
      groups.push_back(k.first);
      plan->angles.push_back(patch_angle_of(ad, bd, t0, k.second));
      plan->A.push_back(std::fabs(a[k.second]));
      plan->B.push_back(std::fabs(b[k.second]));
   }
   plan->segs = patch_runs(groups);
   if (plan->segs.size() > kPatchMaxSegs) return false;
   // symmetric sets: angles i pi / Pp with 0 < i < Pp / 4 stand for four rows each
   if (unrotated && Pp % 2 == 0 && Pp >= 8) {
      groups.clear();
      for (int i = 1; 4 * i < Pp; ++i) {
         groups.push_back(patch_group(a[i], b[i]));
         plan->sym_angles.push_back(patch_angle_of(ad, bd, t0, i));
      }
      plan->sym_segs = patch_runs(groups);
      plan->sym_extra.push_back(patch_angle_of(ad, bd, t0, 0));
      plan->sym_extra.push_back(patch_angle_of(ad, bd, t0, Pp / 2));
      if (Pp % 4 == 0) {  // and its mirror image
         plan->sym_extra.push_back(patch_angle_of(ad, bd, t0, Pp / 4));
         plan->sym_extra.push_back(patch_angle_of(ad, bd, t0, 3 * Pp / 4));
      }
      if (plan->sym_segs.size() > kPatchMaxSegs) plan->sym_angles.clear();
   }
   return true;
}

// Tiles with a pixel inside the inscribed circle (all without a mask), as the
// kernel's test counts them, row by row.
static long live_tiles(int N, bool masked) {
   const int t = (N + kTile - 1) / kTile;
   if (!masked) return (long)t * t;
   const double c = 0.5 * (N - 1), lim = 0.25 * (double)N * N;
   long n = 0;
   for (int r = 0; r < t; ++r) {
      const double y0 = (double)r * kTile, ny = std::max({y0 - c, c - (y0 + kTile - 1), 0.0});
      if (ny * ny > lim) continue;
      const double w = std::sqrt(lim - ny * ny);  // a tile from x0 on meets it if x0 <= c + w and x0 + 15 >= c - w
      const long first = std::max(0L, (long)std::ceil((c - w - (kTile - 1)) / kTile));
      n += std::min((long)t - 1, (long)std::floor((c + w) / kTile)) - first + 1;
   }
   return n;
}

// The rows, then one non-finite flag per quad.
size_t bp_quads_bytes(int batch, int Pp, int Dp) {
   if (batch <= 0) return 0;
   const size_t quads = (size_t)((batch + 3) / 4);
   return sizeof(float4) * quads * Pp * Dp + sizeof(int) * quads;
}

bool bp_patch_rows_ok(const BPCfg& cfg, const float* sino, int batch) {
   return cfg.few && batch <= 2 && cfg.patch && !cfg.patch->angles.empty() && cfg.Dp % 4 == 0 &&
          (reinterpret_cast<uintptr_t>(sino) & 15) == 0;
}

cudaError_t launch_bp_patch(const float* sino, float* img, int batch, const BPCfg& cfg, cudaStream_t st) {
   if (!cfg.patch || cfg.patch->angles.empty() || !cfg.patch_angles || !cfg.err) return cudaErrorInvalidConfiguration;
   PatchPlanParam pp;
   std::memcpy(pp.seg, cfg.patch->segs.data(), sizeof(uint32_t) * cfg.patch->segs.size());
   pp.n_segs = (int)cfg.patch->segs.size();
   cudaError_t e = cudaSuccess;
   if (!cfg.prefilled && bp_patch_rows_ok(cfg, sino, batch)) {
      if (cfg.mid_event && (e = cudaEventRecord(cfg.mid_event, st)) != cudaSuccess) return e;
      RowsArgs r{cfg.patch_angles, sino, img, cfg.err, cfg.N, cfg.Pp, cfg.Dp, 0, cfg.norm, cfg.mask_value, cfg.masking};
      // Groups of angles per CTA: two keep a chunk's refill small beside its work;
      // four where the tiles alone are too few warps (one slice, groups of 2 / 4 /
      // 8: 512^2 119 / 130 / 145 us, 256^2 36 / 28 / 30; with symmetric sets 91 /
      // 99 / 131 and 30 / 27 / 30).
      const bool many = (long)((cfg.N + kTile - 1) / kTile) * ((cfg.N + kTile - 1) / kTile) >= 600;
      if (cfg.part && !cfg.patch->sym_angles.empty()) {
         r.ang = cfg.patch_angles + cfg.patch->angles.size();  // uploaded after the plan's own
         r.img = cfg.part;
         PatchSegs ps;
         std::memcpy(ps.seg, cfg.patch->sym_segs.data(), sizeof(uint32_t) * cfg.patch->sym_segs.size());
         ps.n_segs = (int)cfg.patch->sym_segs.size();
         e = many ? (batch == 1 ? launch_rows<1, 2, true>(r, ps, cfg, st) : launch_rows<2, 2, true>(r, ps, cfg, st))
                  : (batch == 1 ? launch_rows<1, 4, true>(r, ps, cfg, st) : launch_rows<2, 4, true>(r, ps, cfg, st));
         if (e != cudaSuccess) return e;
         CombineArgs ca;
         ca.part = cfg.part;
         ca.sino = sino;
         ca.img = img;
         ca.n_extra = (int)cfg.patch->sym_extra.size();
         for (int i = 0; i < ca.n_extra; ++i) ca.extra[i] = cfg.patch->sym_extra[i];
         ca.N = cfg.N;
         ca.Pp = cfg.Pp;
         ca.Dp = cfg.Dp;
         ca.norm = cfg.norm;
         ca.mask_value = cfg.mask_value;
         ca.masking = cfg.masking;
         const dim3 grid((cfg.N + 31) / 32, (cfg.N + 7) / 8);
         if (batch == 1) bp_patch_combine<1><<<grid, 256, 0, st>>>(ca);
         else bp_patch_combine<2><<<grid, 256, 0, st>>>(ca);
         return cudaGetLastError();
      }
      if (many)
         return batch == 1 ? launch_rows<1, 2, false>(r, pp, cfg, st) : launch_rows<2, 2, false>(r, pp, cfg, st);
      return batch == 1 ? launch_rows<1, 4, false>(r, pp, cfg, st) : launch_rows<2, 4, false>(r, pp, cfg, st);
   }
   if (!cfg.pairs || bp_quads_bytes(batch, cfg.Pp, cfg.Dp) > cfg.pairs_bytes) return cudaErrorInvalidValue;
   std::memcpy(pp.A, cfg.patch->A.data(), sizeof(float) * cfg.Pp);
   std::memcpy(pp.B, cfg.patch->B.data(), sizeof(float) * cfg.Pp);
   const int nq = (batch + 3) / 4;
   float4* quads = static_cast<float4*>(cfg.pairs);
   int* flags = reinterpret_cast<int*>(quads + (size_t)nq * cfg.Pp * cfg.Dp);
   PatchArgs a;
   a.ang = cfg.patch_angles;
   a.nonfinite = cfg.prefilled ? nullptr : flags;  // the engine's rows are finite: logarithms of clamped counts
   a.quads = quads;
   a.img = img;
   a.err = cfg.err;
   a.N = cfg.N;
   a.Pp = cfg.Pp;
   a.Dp = cfg.Dp;
   a.batch = batch;
   a.n_quads = nq;
   a.norm = cfg.norm;
   a.mask_value = cfg.mask_value;
   a.masking = cfg.masking;
   if (!cfg.prefilled) {
      if ((e = cudaMemsetAsync(flags, 0, sizeof(int) * nq, st)) != cudaSuccess) return e;
      bp_quads_fill<<<dim3((cfg.Dp + 255) / 256, cfg.Pp, nq), 256, 0, st>>>(sino, quads, flags, batch, cfg.Pp, cfg.Dp);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
   }
   if (cfg.mid_event && (e = cudaEventRecord(cfg.mid_event, st)) != cudaSuccess) return e;
   // Slice quads per thread (SQ) and per load phase (QL) by the batch and the
   // bins per pixel. Up to 1.25 bins per pixel the neighbouring patches of a
   // phase fall in different banks as they are, so few quads per phase do as
   // well as eight and leave smaller CTAs: 16 slices of 1024^2 at 1 bin per pixel
   // 2.19 ms with (2, 2), 2.77 with (1, 4). Above, patches collide (64 slices at
   // 1.5: (2, 2) 2.35 ms, (2, 8) 1.72) and a phase takes more quads. All forms add
   // the same terms in the same order: same bits.
   if (nq == 1) return launch_patch<1, 1, 10>(a, pp, cfg.scale, st);
   if (nq == 2) return launch_patch<1, 2, 6>(a, pp, cfg.scale, st);
   // The larger forms cost less per slice but leave more of the SMs idle at the end:
   // the most CTAs that an SM gets, of the tiles that meet the circle where it is
   // masked, times a form's cost.
   const long live = live_tiles(cfg.N, cfg.masking != 0);
   auto rounds = [live, nq](int quads) { return (live * ((nq + quads - 1) / quads) + kSMs - 1) / kSMs; };
   if (cfg.scale <= 1.25f) {
      // Four quads per thread spread a patch's weights (a fifth of the FP32 work)
      // over twice the slices: 1.84 times the time of half the slices (32 slices of
      // 512^2 x 720 angles 773 us against 844, of 256^2 x 512 128 slices 570 against 618;
      // 64 slices of that, four CTAs per SM for seven halves, 217 against 209), if an SM
      // has two.
      if (live * ((nq + 7) / 8) >= 2 * kSMs && 184 * rounds(8) <= 100 * rounds(4))
         return launch_patch<4, 2, 2>(a, pp, cfg.scale, st);
      return launch_patch<2, 2, 3>(a, pp, cfg.scale, st);
   }
   if (nq <= 4) return launch_patch<1, 4, 3>(a, pp, cfg.scale, st);
   // The CTA of 16 quads shares a pixel's weights between twice the slices of 8 quads:
   // 1.65 times the time of 8 quads (2.11 against 1.25 ms, 512^2 x 1024 angles; 60
   // slices of 256^2 x 512, two for four, 398 us against 456, but for three, masked, 397
   // against 356). That of 4 quads takes 0.6 of it, 0.53 up to 1.5 bins per pixel (30 masked
   // slices of 256^2: 199 and 220 us at 1.5 and 2 bins, with 8 240 and 242; 64 slices of
   // 128^2 at 2: one of 8 quads 80 us, two of 4 89, one of 16 119).
   const long c4 = (cfg.scale <= 1.5f ? 53 : 60) * rounds(4), c8 = 100 * rounds(8), c16 = 165 * rounds(16);
   if (c16 <= c8 && c16 <= c4) return launch_patch<2, 8, 1, true>(a, pp, cfg.scale, st);
   if (c4 < c8) return launch_patch<1, 4, 3>(a, pp, cfg.scale, st);
   // Two CTAs of 8 quads per SM (their registers held to 56, a few spilled) hide each
   // other's waits, 30 slices of 512^2 1484 us against 1531; a CTA that has its SM to
   // itself is faster without (20 masked slices of 200^2 129 us against 190).
   return rounds(8) > 1 ? launch_patch<1, 8, 2>(a, pp, cfg.scale, st) : launch_patch<1, 8, 1>(a, pp, cfg.scale, st);
}
}  // namespace risa_gb
