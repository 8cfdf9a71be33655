// Sub-bucket construction for stride-S pooling, sm_100a.
//
// Replaces local_subbuck_ker (src/psh/batch_psh_subbuck_reduce.cuh:104-298) and its CumsumCounter
// (src/psh/shmem_cumsum_counter.cuh:25-167).  Per 1024-point block of a scene:
//   block bounding box -> block-normalised voxel -> 13-bit key (16-bit hash / 8, 8192 bins, :130-131,202-203)
//   -> points ordered by (key, index) -> runs of S consecutive points form one sub-bucket
//   -> subbuck_id / subbuck_off / unpool_ind[row, off] = global row, reduced_coord[row] = mean of member coords.
//
// Deliberate, documented differences from the reference, all of which remove run-to-run variation:
//   * no random rotation before the bounding box (the reference draws a fresh quaternion per launch, :193-195);
//   * the block bounding box is the true min/max, broadcast to every thread (the reference consumes a
//     cub::BlockReduce result that is only defined in thread 0, src/common/block_minmax.cuh:43-47);
//   * equal keys are ordered by input index (the reference: shared-memory atomic arrival order);
//   * block k of a scene owns rows [k*ceil(1024/S), ...) of the scene's reduced rows (the reference hands out
//     row ranges with a global atomicAdd in block arrival order, :238);
//   * coordinate means are summed sequentially in sub-bucket order in fp32 (the reference: float shared-memory
//     atomics, :261-270), so the result is bit-reproducible.
#include "f3d_common.cuh"
#include "psh_device.cuh"
#include "../../include/f3d_b200.h"

namespace f3d {

constexpr uint32_t kSbPoints = 1024;          // points of a block (the reference's block)
constexpr uint32_t kSbBins = 8192;
constexpr uint32_t kSbSegDiv = 65536 / kSbBins;
constexpr uint32_t kSbVecs = kSbBins / 8;     // 128-bit words of the bins, 16 bits a bin
constexpr uint32_t kSbCrowd = 32;             // a bin of more points orders them with a bit mask
constexpr uint32_t kSbCrowds = kSbPoints / (kSbCrowd + 1);

struct SubbuckArgs {
  const __half *coord; const uint32_t *batch_sep; const uint32_t *red_sep;
  uint32_t *subbuck_id; uint16_t *subbuck_off; uint32_t *unpool_ind; __half *reduced_coord;
  uint32_t total_N, batch, S, num_vox, hash_type, red_rows /* rows of unpool_ind */, red_coord_rows;
};

// fp16 values in the order of unsigned integers (the sign bit is the top bit of 16), and back
__device__ __forceinline__ uint32_t half_order(float v) {
  const uint32_t u = __half_as_ushort(__float2half_rn(v));      // v is an fp16 value: exact
  return u & 0x8000u ? 0xFFFFu ^ u : u | 0x8000u;
}
__device__ __forceinline__ float half_from_order(uint32_t k) {
  return __half2float(__ushort_as_half((unsigned short)(k & 0x8000u ? k ^ 0x8000u : 0xFFFFu ^ k)));
}

// PER points a thread, 1024 / PER threads.  Bound by barriers, shared-memory passes and warp reductions, not by the 16 bytes a
// point moves, so: the bins are 16-bit (a block has 1024 points), which makes zeroing, scanning and writing back 8192 of them
// one conflict-free 128-bit pass each; the box is reduced by redux on order-preserving integers instead of shuffles; a voxel
// index takes the division-free form of vox_axis; unpool_ind leaves in order of its own rows instead of scattered.  Points of
// one bin are ordered by counting the smaller indices among them, which is quadratic in the bin: a crowded bin (many points of
// one voxel) takes a 1024-bit mask of its members instead, with the population of the words in front.
// Three levels of 8 x 1M points with heavy-tailed voxels: 717 us with one point a thread, 32-bit bins and the count for every
// bin; 393 us without the masks; 239 us now.
template <uint32_t PER>
__global__ void __launch_bounds__(kSbPoints / PER, PER == 1 ? 1 : 4) subbuck_build_kernel(SubbuckArgs a) {
  constexpr uint32_t kThreads = kSbPoints / PER, kWarps = kThreads / 32;
  constexpr uint32_t kVecs = kSbVecs / kWarps;                // 128-bit words of the bins that a warp scans
  __shared__ __align__(16) uint16_t bins[kSbBins];            // counts, then first positions; later the members in order:
  uint2 *const member = reinterpret_cast<uint2 *>(bins);      // [1024] coordinates (x | y, z) and index in the block, by position,
  uint16_t *const crowd_pre = bins + kSbBins / 2;             // and [kSbCrowds][32] members in front of each mask word
  __shared__ uint16_t sorted_ind[kSbPoints];                  // members of a bin as they came; of a crowded bin its mask's number
  __shared__ uint32_t crowd_mask[kSbCrowds][32];
  __shared__ uint32_t box[6], crowds;
  __shared__ uint32_t wsum[kWarps];

  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (uint32_t i = 0; i < kSbVecs / kThreads; ++i) reinterpret_cast<uint4 *>(bins)[tid + i * kThreads] = make_uint4(0u, 0u, 0u, 0u);
  for (uint32_t i = tid; i < kSbCrowds * 32; i += kThreads) (&crowd_mask[0][0])[i] = 0u;
  if (tid < 6) box[tid] = tid < 3 ? 0xFFFFu : 0u;
  if (tid == 6) crowds = 0u;
  grid_enter();
  const uint32_t scene = blockIdx.y;
  // alignment rows behind the reduced rows
  if (blockIdx.x == 0 && scene == 0)
    for (uint64_t i = (uint64_t)a.red_rows * 3 + tid; i < (uint64_t)a.red_coord_rows * 3; i += kThreads) a.reduced_coord[i] = __float2half_rn(0.f);
  const uint32_t start = scene ? a.batch_sep[scene - 1] : 0u;
  const uint32_t end = min(a.batch_sep[scene], a.total_N);
  const uint32_t n = end > start ? end - start : 0u;
  const uint32_t blk0 = blockIdx.x * kSbPoints;
  if (blk0 >= n) return;
  const uint32_t pts = min(kSbPoints, n - blk0);
  const uint32_t red_start = scene ? a.red_sep[scene - 1] : 0u;
  const uint32_t red_end = a.red_sep[scene];
  const uint32_t g0 = start + blk0;

  float c[PER][3];
#pragma unroll
  for (uint32_t i = 0; i < PER; ++i) {
    const uint32_t p = tid + i * kThreads;
#pragma unroll
    for (int d = 0; d < 3; ++d) c[i][d] = p < pts ? __half2float(a.coord[(size_t)(g0 + p) * 3 + d]) : 0.f;
  }
  __syncthreads();                                             // bins, masks and box are set
  // box of the block's points; a NaN coordinate takes no part
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float lo = INFINITY, hi = -INFINITY;
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i)
      if (tid + i * kThreads < pts) { lo = fminf(lo, c[i][d]); hi = fmaxf(hi, c[i][d]); }
    const uint32_t l = __reduce_min_sync(0xFFFFFFFFu, half_order(lo)), h = __reduce_max_sync(0xFFFFFFFFu, half_order(hi));
    if (lane == 0) { atomicMin(&box[d], l); atomicMax(&box[3 + d], h); }
  }
  __syncthreads();
  uint32_t key[PER], at[PER];                                  // at: order of arrival in the bin
  {
    uint32_t v[PER][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float lo = half_from_order(box[d]), hi = half_from_order(box[3 + d]);
      const AxisScale ax = make_axis_scale(lo, hi, a.num_vox);
      if (ax.r != 0.f) {
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) v[i][d] = vox_axis(c[i][d], ax);
      } else {                                                 // an infinite extent
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) v[i][d] = vox_axis(c[i][d], lo, hi, a.num_vox);
      }
    }
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) {
      switch (a.hash_type) {
        case H_ZORDER_DIV: key[i] = zorder16(v[i][0], v[i][1], v[i][2]) / kSbSegDiv; break;
        case H_XORSUM_DIV: key[i] = ((v[i][0] ^ v[i][1] ^ v[i][2]) & 0xFFFFu) / kSbSegDiv; break;
        case H_ZORDER_MOD: key[i] = zorder16(v[i][0], v[i][1], v[i][2]) % kSbBins; break;
        default:           key[i] = ((v[i][0] ^ v[i][1] ^ v[i][2]) & 0xFFFFu) % kSbBins; break;
      }
      at[i] = 0;
      if (tid + i * kThreads < pts) {
        const uint32_t sh = (key[i] & 1u) * 16u;
        at[i] = (atomicAdd(reinterpret_cast<uint32_t *>(bins) + (key[i] >> 1), 1u << sh) >> sh) & 0xFFFFu;
      }
    }
  }
  __syncthreads();
  // exclusive scan of the bins: a warp takes kVecs words of eight, 32 words a step
  {
    uint4 *const vec = reinterpret_cast<uint4 *>(bins) + warp * kVecs + lane;
    uint32_t ex[kVecs / 32], carry = 0;
#pragma unroll
    for (uint32_t j = 0; j < kVecs / 32; ++j) {
      const uint4 w = vec[j * 32];
      const uint32_t pair = w.x + w.y + w.z + w.w, sum = (pair & 0xFFFFu) + (pair >> 16);
      uint32_t inc = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, inc, d);
        if (lane >= d) inc += o;
      }
      ex[j] = carry + inc - sum;
      carry += __shfl_sync(0xFFFFFFFFu, inc, 31);
    }
    if (lane == 0) wsum[warp] = carry;
    __syncthreads();
    const uint32_t front = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? wsum[lane] : 0u);
#pragma unroll
    for (uint32_t j = 0; j < kVecs / 32; ++j) {
      uint4 w = vec[j * 32];
      uint32_t run = front + ex[j];
      uint32_t *e = reinterpret_cast<uint32_t *>(&w);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t lo = e[q] & 0xFFFFu, hi = e[q] >> 16;
        e[q] = run | ((run + lo) << 16);
        run += lo + hi;
      }
      vec[j * 32] = w;
    }
  }
  __syncthreads();
  uint32_t base[PER], cnt[PER];
#pragma unroll
  for (uint32_t i = 0; i < PER; ++i) {
    const uint32_t p = tid + i * kThreads;
    base[i] = cnt[i] = 0;
    if (p < pts) {
      base[i] = bins[key[i]];
      cnt[i] = (key[i] + 1 < kSbBins ? (uint32_t)bins[key[i] + 1] : pts) - base[i];
      if (cnt[i] <= kSbCrowd) sorted_ind[base[i] + at[i]] = (uint16_t)p;
      else if (at[i] == 0) sorted_ind[base[i]] = (uint16_t)atomicAdd(&crowds, 1u);
    }
  }
  __syncthreads();
  if (crowds) {
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) {                       // a warp's 32 points of a step are the 32 bits of one word
      const uint32_t slot = cnt[i] > kSbCrowd ? sorted_ind[base[i]] : kSbCrowds;
      const uint32_t peers = __match_any_sync(0xFFFFFFFFu, slot);
      if (slot < kSbCrowds && (peers & ((1u << lane) - 1u)) == 0u) crowd_mask[slot][i * kWarps + warp] = peers;
    }
    __syncthreads();
    for (uint32_t s = warp; s < crowds; s += kWarps) {
      const uint32_t pop = __popc(crowd_mask[s][lane]);
      uint32_t inc = pop;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, inc, d);
        if (lane >= d) inc += o;
      }
      crowd_pre[s * 32 + lane] = (uint16_t)(inc - pop);
    }
    __syncthreads();
  }
  const uint32_t per_block = (kSbPoints + a.S - 1) / a.S;
  const uint32_t row0 = blockIdx.x * per_block;               // first reduced row of the block in its scene
#pragma unroll
  for (uint32_t i = 0; i < PER; ++i) {
    const uint32_t p = tid + i * kThreads;
    if (p < pts) {
      uint32_t pos = base[i];
      if (cnt[i] > kSbCrowd) {
        const uint32_t s = sorted_ind[base[i]], w = i * kWarps + warp;
        pos += crowd_pre[s * 32 + w] + __popc(crowd_mask[s][w] & ((1u << lane) - 1u));
      } else if (cnt[i] > 1) {
        for (uint32_t j = 0; j < cnt[i]; ++j) pos += sorted_ind[base[i] + j] < p ? 1u : 0u;
      }
      const uint32_t sub = pos / a.S;
      a.subbuck_id[g0 + p] = row0 + sub;
      a.subbuck_off[g0 + p] = (uint16_t)(pos - sub * a.S);
      const uint32_t x = __half_as_ushort(__float2half_rn(c[i][0])), y = __half_as_ushort(__float2half_rn(c[i][1])),
                     z = __half_as_ushort(__float2half_rn(c[i][2]));
      member[pos] = make_uint2(x | (y << 16), z | (p << 16));
    }
  }
  __syncthreads();
  // members row by row; the last sub-bucket of a block may be short: its unfilled slots take the out-of-range index the
  // reference pre-fills the whole table with (flash3dxfmr/psh/subbuck.py:94), so the table needs no pre-fill
  const uint32_t first = red_start + row0;
  const uint32_t stop = min(red_end, a.red_rows);
  const uint32_t rows = first < stop ? min((pts + a.S - 1) / a.S, stop - first) : 0u;
  uint32_t *const out = a.unpool_ind + (size_t)first * a.S;
  for (uint32_t p = tid; p < rows * a.S; p += kThreads) out[p] = p < pts ? g0 + (member[p].y >> 16) : a.total_N + 3u;
  const uint32_t crows = first < a.red_coord_rows ? min(rows, a.red_coord_rows - first) : 0u;
  for (uint32_t r = tid; r < crows; r += kThreads) {
    const uint32_t p0 = r * a.S, m = min(a.S, pts - p0);
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
    for (uint32_t j = 0; j < m; ++j) {
      const uint2 w = member[p0 + j];
      const float x = __half2float(__ushort_as_half((unsigned short)(w.x & 0xFFFFu))), y = __half2float(__ushort_as_half((unsigned short)(w.x >> 16))),
                  z = __half2float(__ushort_as_half((unsigned short)(w.y & 0xFFFFu)));
      s0 = j ? __fadd_rn(s0, x) : x; s1 = j ? __fadd_rn(s1, y) : y; s2 = j ? __fadd_rn(s2, z) : z;
    }
    const float cntf = (float)m;
    __half *const o = a.reduced_coord + (size_t)(first + r) * 3;
    o[0] = __float2half_rn(__fdiv_rn(s0, cntf));
    o[1] = __float2half_rn(__fdiv_rn(s1, cntf));
    o[2] = __float2half_rn(__fdiv_rn(s2, cntf));
  }
}

int subbuck_build(const void *coord, const void *batch_sep, const void *red_sep, void *subbuck_id, void *subbuck_off,
                  void *unpool_ind, void *reduced_coord, uint32_t total_N, uint32_t batch, uint32_t max_n, uint32_t S,
                  uint32_t num_vox, uint32_t hash_type, uint32_t red_rows, uint32_t red_coord_rows, int device, cudaStream_t st) {
  SubbuckArgs a{};
  a.coord = static_cast<const __half *>(coord);
  a.batch_sep = static_cast<const uint32_t *>(batch_sep);
  a.red_sep = static_cast<const uint32_t *>(red_sep);
  a.subbuck_id = static_cast<uint32_t *>(subbuck_id);
  a.subbuck_off = static_cast<uint16_t *>(subbuck_off);
  a.unpool_ind = static_cast<uint32_t *>(unpool_ind);
  a.reduced_coord = static_cast<__half *>(reduced_coord);
  a.total_N = total_N; a.batch = batch; a.S = S; a.num_vox = num_vox; a.hash_type = hash_type;
  a.red_rows = red_rows; a.red_coord_rows = red_coord_rows;
  const bool any = max_n > 0 && batch > 0;
  if (any) {
    // Few blocks leave SMs idle: a thread a point then gives the shorter chain (four levels of a 20,000-point scan: 37 us
    // against 71); past one block an SM, four points a thread keep more blocks on each.
    const dim3 grid(cdiv_u32(max_n, kSbPoints), batch);
    if ((uint64_t)grid.x * batch <= (uint64_t)sm_count(device)) launch(subbuck_build_kernel<1>, grid, kSbPoints, 0, st, a);
    else launch(subbuck_build_kernel<4>, grid, kSbPoints / 4, 0, st, a);
  } else if (red_coord_rows > red_rows) {
    F3D_CUDA_TRY(cudaMemsetAsync(a.reduced_coord + (size_t)red_rows * 3, 0, (size_t)(red_coord_rows - red_rows) * 6, st));
  }
  return check_launch("subbuck_build", any ? 1 : 0);
}

}  // namespace f3d
