// Bounding box of fp16 coordinates [N, 3]: the minimum and maximum over all rows that the reference takes with
// coords.min(0) / coords.max(0) before every bucketing (flash3dxfmr/psh/psh_main.py:117-118).  A NaN in a column makes both of
// its ends NaN, as torch does.
//
// Bound by HBM for large batches (6 bytes per point read once), by the launch for one scan.  A thread takes eight points as
// three 16-byte loads: the twelve packed pairs of such a group repeat the components (x,y) (z,x) (y,z), so three packed
// accumulators hold everything and a point costs three packed minima and maxima.  Up to kOneBlockPoints one block does it
// all; above, one row of partial results per block and a second launch of one block.  (A column reduction of the general
// kind takes 23 us for 20,000 points and 40 us for 1.9 M.)
#include "f3d_common.cuh"
#include "../../include/f3d_b200.h"

namespace f3d {

constexpr int kBoxThreads = 512;
constexpr uint32_t kOneBlockPoints = 1u << 15;      // 192 KB: below that the second launch costs more than the idle SMs
constexpr uint32_t kBoxBlocks = 296;                // two blocks per SM

struct Box3 {
  __half2 lo[3], hi[3];                             // pairs (x, y) (z, x) (y, z)
};

__device__ __forceinline__ void box_init(Box3 &b) {
  const __half2 inf = __half2half2(__ushort_as_half(0x7C00)), ninf = __half2half2(__ushort_as_half(0xFC00));
#pragma unroll
  for (int i = 0; i < 3; ++i) { b.lo[i] = inf; b.hi[i] = ninf; }
}
__device__ __forceinline__ void box_add(Box3 &b, int i, __half2 v) {
  b.lo[i] = __hmin2_nan(b.lo[i], v);
  b.hi[i] = __hmax2_nan(b.hi[i], v);
}

// the box of the block's points (written by thread 0 as min x, y, z, max x, y, z)
__device__ __forceinline__ void box_store(Box3 b, __half *lo, __half *hi) {
  __shared__ Box3 part[kBoxThreads / 32];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int d = 16; d; d >>= 1) {
      b.lo[i] = __hmin2_nan(b.lo[i], __shfl_xor_sync(0xFFFFFFFFu, b.lo[i], d));
      b.hi[i] = __hmax2_nan(b.hi[i], __shfl_xor_sync(0xFFFFFFFFu, b.hi[i], d));
    }
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < kBoxThreads / 32; ++w)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      b.lo[i] = __hmin2_nan(b.lo[i], part[w].lo[i]);
      b.hi[i] = __hmax2_nan(b.hi[i], part[w].hi[i]);
    }
  lo[0] = __hmin_nan(__low2half(b.lo[0]), __high2half(b.lo[1]));
  lo[1] = __hmin_nan(__high2half(b.lo[0]), __low2half(b.lo[2]));
  lo[2] = __hmin_nan(__low2half(b.lo[1]), __high2half(b.lo[2]));
  hi[0] = __hmax_nan(__low2half(b.hi[0]), __high2half(b.hi[1]));
  hi[1] = __hmax_nan(__high2half(b.hi[0]), __low2half(b.hi[2]));
  hi[2] = __hmax_nan(__low2half(b.hi[1]), __high2half(b.hi[2]));
}

// VEC: the coordinates start on a 16-byte boundary.  Block b of `gridDim.x` leaves its box at lo + 6 b, hi + 6 b.
template <bool VEC>
__global__ void __launch_bounds__(kBoxThreads) bbox_kernel(const __half *__restrict__ c, uint32_t n, __half *lo, __half *hi) {
  const uint32_t after = grid_enter();
  c += after;
  Box3 b;
  box_init(b);
  const uint32_t stride = gridDim.x * kBoxThreads, first = blockIdx.x * kBoxThreads + threadIdx.x;
  uint32_t done = 0;
  if (VEC) {
    const uint4 *c4 = reinterpret_cast<const uint4 *>(c);
    const uint32_t groups = n / 8;
    for (uint32_t g = first; g < groups; g += stride) {
      const uint4 q[3] = {__ldg(c4 + 3 * (size_t)g), __ldg(c4 + 3 * (size_t)g + 1), __ldg(c4 + 3 * (size_t)g + 2)};
      const __half2 *h = reinterpret_cast<const __half2 *>(q);
#pragma unroll
      for (int i = 0; i < 12; ++i) box_add(b, i % 3, h[i]);
    }
    done = groups * 8;
  }
  for (uint32_t r = done + first; r < n; r += stride) {
    const __half *p = c + 3 * (size_t)r;
    const __half x = p[0], y = p[1], z = p[2];
    box_add(b, 0, __halves2half2(x, y));
    box_add(b, 1, __halves2half2(z, x));
    box_add(b, 2, __halves2half2(y, z));
  }
  box_store(b, lo + 6 * (size_t)blockIdx.x, hi + 6 * (size_t)blockIdx.x);
}

__global__ void __launch_bounds__(kBoxThreads) bbox_final_kernel(const __half *__restrict__ part, uint32_t blocks, __half *lo, __half *hi) {
  const uint32_t after = grid_enter();
  part += after;
  Box3 b;
  box_init(b);
  for (uint32_t r = threadIdx.x; r < blocks; r += kBoxThreads) {
    const __half *p = part + 6 * (size_t)r;
    b.lo[0] = __hmin2_nan(b.lo[0], __halves2half2(p[0], p[1]));
    b.lo[1] = __hmin2_nan(b.lo[1], __halves2half2(p[2], p[0]));
    b.lo[2] = __hmin2_nan(b.lo[2], __halves2half2(p[1], p[2]));
    b.hi[0] = __hmax2_nan(b.hi[0], __halves2half2(p[3], p[4]));
    b.hi[1] = __hmax2_nan(b.hi[1], __halves2half2(p[5], p[3]));
    b.hi[2] = __hmax2_nan(b.hi[2], __halves2half2(p[4], p[5]));
  }
  box_store(b, lo, hi);
}

}  // namespace f3d

using namespace f3d;

extern "C" int f3d_bbox_f16(const void *coords, void *bbox_min, void *bbox_max, uint32_t rows, int device, void *stream) {
  if (rows == 0) return set_error(F3D_ERR_ARG, "bbox: no points");
  DeviceGuard guard(device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const __half *c = static_cast<const __half *>(coords);
  __half *lo = static_cast<__half *>(bbox_min), *hi = static_cast<__half *>(bbox_max);
  const bool vec = reinterpret_cast<uintptr_t>(coords) % 16 == 0;
  const bool one = rows <= kOneBlockPoints;
  __half *out_lo = lo, *out_hi = hi;
  uint32_t blocks = 1;
  if (!one) {
    blocks = cdiv_u32(rows, 8 * kBoxThreads);
    if (blocks > kBoxBlocks) blocks = kBoxBlocks;
    void *part = nullptr;
    F3D_TRY(workspace(device, 8, kBoxBlocks * 6 * sizeof(__half), st, &part));
    out_lo = static_cast<__half *>(part);
    out_hi = out_lo + 3;
  }
  if (vec) launch(bbox_kernel<true>, blocks, kBoxThreads, 0, st, c, rows, out_lo, out_hi);
  else launch(bbox_kernel<false>, blocks, kBoxThreads, 0, st, c, rows, out_lo, out_hi);
  if (!one) launch(bbox_final_kernel, 1, kBoxThreads, 0, st, out_lo, blocks, lo, hi);
  F3D_TRY(check_launch("bbox", one ? 1 : 2));
  return maybe_sync(st, "bbox");
}
