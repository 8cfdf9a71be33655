// Bucketed self-attention backward on tcgen05 tensor cores, sm_100a.
//
// Implements buck_swin_bwd(Q, K, V, O, dO, LSE, Delta, dQ, dK, dV, Scope_buckets, bucket_size), which the reference's
// Python layer calls (flash3dxfmr/layers/buck_swin.py:91) but whose kernel and binding are absent from the reference
// snapshot (declaration src/f3d_frontend.cu:94-97, binding commented out :137).  Semantics follow the reference's
// tests (tests/test_attn_bwd.py:24-27,54-62,79-441): Delta[b,t,h] = sum_d dO*O is written to the caller's buffer;
// with P = exp(S - LSE), dV = P^T dO, dP = dO V^T, dS = P o (dP - Delta), dQ = dS K / sqrt(D), dK = dS^T Q / sqrt(D).
// O and LSE may come from any forward implementation (the tests pass FlashAttention's).
//
// Kernels:
//   attn_bwd_delta_kernel   Delta = rowsum(dO o O), one thread per (token, head)
//   attn_bwd_kernel<D>      one CTA per (scope, 128-key block, head, batch row); it loops over the query tiles of the
//                           scope and keeps dK, dV for its keys in tensor memory.  D = 64 / 128: one CTA per SM with 512
//                           tensor-memory columns.  D <= 32 (32 is the backbone's head size): TWO CTAs per SM with 256
//                           columns each and 64-query tiles, so that one CTA computes while the other waits
//       producer    TMA: K_j, V_j once; Q_i, dO_i through a 2- or 3-stage ring
//       MMA warp    issues S^T = K Q^T and dP^T = V dO^T into tensor memory (keys on the lanes); -lse and -delta of the
//                   queries ride in them as an extra k-step (BwdCfg::kOnesBytes).  Once the compute warps hold tile i in
//                   registers it issues those products of tile i + 1, and once they have published P^T and dS^T
//                   dV += P^T dO and dK += dS^T Q (P^T from tensor memory where the columns allow it, else K-major
//                   shared-memory tiles) and dQ_i = dS K (the dS^T tile read as an MN-major A operand)
//       compute     P^T = exp2(S^T c), dS^T = P^T o dP^T, both as bf16; then the dQ tile of the iteration before: into the
//                   fp32 scratch with vector reductions, or (D = 32) through shared memory and
//       drain warp  (D = 32) one thread hands each staged dQ tile to the copy engine as a single add-reduce
//                   (cp.reduce.async.bulk.tensor) and recycles the two staging buffers
//       constants   the rows of the extra k-step, a ring stage ahead
//   attn_bwd_dq_convert     dQ = bf16(scratch / sqrt(D))
// dQ needs the scratch because every key block of a scope contributes to every query; dK and dV are written once.
//
// What bounds it (D = 32): the chain of one tile, 2,200 cycles with two CTAs on the SM, of which the compute warps work all
// but 200; the shared-memory pipe and the schedulers are two thirds busy.  What took it there (B200, W = 4096, TFLOP/s):
// score products issued as soon as the tile before is in registers, descriptors as a base and constant steps, half the
// barriers 485 -> 505; the per-query constants on a warp of their own instead of two of the compute warps 505 -> 585
// (D = 16: 265 -> 286 -> 300); lanes without a query leave the dQ staging to the others 585 -> 600.  D = 64 / 128: no
// change (525 / 550-600).  Measured and not kept: the dQ products of two 64-query tiles as one M = 128 product (its operand
// reads halve, but tile i + 2 then waits for it: 585 -> 536).  Windows of up to 512 tokens had a kernel of their own that
// kept every dQ tile in tensor memory; this one is faster there now (W = 512: 336 -> 370, W = 256: 233 -> 239).
#include "f3d_common.cuh"
#include "tc_sm100.cuh"
#include "../../include/f3d_b200.h"

namespace f3d {

int *status_word(int device);

constexpr int kBK = 128;               // keys per CTA (tensor-memory lanes)

struct AttnBwdArgs {
  const float *lse; const float *delta; float *dq_acc; __nv_bfloat16 *dK; __nv_bfloat16 *dV; const uint32_t *scopes;
  int B, L, H, num_scopes, k, bucket, kblocks_per_bucket;
  float scale_log2, scale, inv_scale;       // log2(e) / sqrt(D), 1 / sqrt(D), sqrt(D)
  int *status;
};

__device__ __forceinline__ float bwd_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// packed fp32 pairs
__device__ __forceinline__ uint64_t bpack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void bunpack2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t bmul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <int D> struct BwdCfg {
  // D <= 32 (32 is the backbone's head size) runs as TWO CTAs per SM: tiles of 64 queries, eight compute warps and 256
  // tensor-memory columns per CTA.  A CTA's tile is a chain of hand-offs (score products -> compute warps -> gradient
  // products -> dQ read-out) in which the compute warps, the busiest part, work less than half of the time; with two
  // CTAs on the SM one computes while the other waits.
  static constexpr bool kTwo = D <= 32;
  static constexpr int kMinCtas = kTwo ? 2 : 1;
  static constexpr int kCW = kTwo ? 8 : 16;        // compute warps: kCW / 4 per tensor-memory lane quadrant
  static constexpr int BQ = (D == 128 || kTwo) ? 64 : 128;       // queries per inner tile
  static constexpr int QCOLS = BQ / (kCW / 4);                   // query columns per compute thread
  static constexpr int kChunk = kTwo ? 16 : QCOLS;               // of which are held in registers at a time
  static constexpr int DCH = D < 64 ? D : 64;
  static constexpr int NDCH = D / DCH;
  static constexpr int RB = DCH * 2;
  static constexpr uint64_t SWZ = RB == 128 ? tc::kSwizzle128 : (RB == 64 ? tc::kSwizzle64 : tc::kSwizzle32);
  static constexpr int kKVBytes = kBK * D * 2;                   // one of K_j, V_j
  static constexpr int kQBytes = BQ * D * 2;                     // one of Q_i, dO_i
  static constexpr int kQStage = 2 * kQBytes;
  static constexpr int QS = D <= 32 ? 3 : 2;                     // Q / dO stages
  static constexpr int PB = D == 64 ? 1 : 2;                     // P^T / dS^T shared-memory buffers (what fits in 227 KB)
  static constexpr int kPBytes = kBK * BQ * 2;                   // P^T or dS^T tile
  // With D <= 32 the bf16 P^T tile also fits in tensor memory: dV then takes its A operand from there and only dS^T, which
  // dQ = dS K reads transposed, goes through shared memory.
  static constexpr bool kTS = D <= 32;
  static constexpr int kBufBytes = kTS ? kPBytes : 2 * kPBytes;  // per buffer: dS^T (| P^T)
  // -lse and -delta enter the score products themselves.  S^T = K Q^T gets one more k-step of 16 whose K side is a constant
  // tile of ones and whose Q side holds -lse * sqrt(D) of each query as three bf16 terms (hi + mid + lo, exact to 2^-24), so
  // the product comes out as s - lse / scale; dP^T = V dO^T likewise comes out as dp - delta.  Otherwise every compute thread
  // has to fetch both constants for each of its columns from shared memory: broadcast loads that cost a wavefront per value
  // and warp and were a third of all shared-memory traffic.
  static constexpr int kOnesBytes = kBK * 32;                      // [128 keys][16] bf16, ones in three columns of each half
  static constexpr int kXBytes = BQ * 32;                          // [BQ queries][16] bf16: the three terms, then zeros
  // D = 32: the dQ tile (128 rows of 128 bytes) leaves through shared memory and ONE add-reduce of the copy engine
  // instead of 1024 vector reductions issued by the compute warps; two staging buffers
  static constexpr bool kTmaDq = D == 32;
  static constexpr int kDqStageBytes = kTmaDq ? BQ * D * 4 : 0;
  static constexpr int kSmem = 2 * kKVBytes + QS * kQStage + PB * kBufBytes + 2 * kDqStageBytes + kOnesBytes + QS * 2 * kXBytes +
                               256 + 1024;
  // producer, MMA, compute warps, one warp for the per-query constants and one that feeds the copy engine (kTmaDq)
  static constexpr int kConstWarp = 2 + kCW, kDrainWarp = kConstWarp + 1;
  static constexpr int kThreads = 32 * (kDrainWarp + (kTmaDq ? 1 : 0));
  static_assert(kSmem <= 227 * 1024, "shared memory budget");
  // tensor-memory columns: S^T, dP^T, (P^T, dS^T as bf16 pairs), dV, dK, dQ
  static constexpr uint32_t kSCol = 0, kDpCol = BQ, kPtCol = 2 * BQ;
  static constexpr uint32_t kDvCol = kTS ? 2 * BQ + BQ / 2 : 2 * BQ, kDkCol = kDvCol + D, kDqCol = kDkCol + D;
  static constexpr uint32_t kTmemCols = kTwo ? 256 : 512;
  static_assert(kDqCol + D <= kTmemCols, "tensor-memory budget");
};

template <int D>
__global__ void __launch_bounds__(BwdCfg<D>::kThreads, BwdCfg<D>::kMinCtas)
attn_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                const __grid_constant__ CUtensorMap map_dq, AttnBwdArgs a) {
  using C = BwdCfg<D>;
  constexpr int BQ = C::BQ, QS = C::QS, PB = C::PB;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *sk = smem, *sv = sk + C::kKVBytes;
  unsigned char *sqdo = sv + C::kKVBytes;                         // [QS stages][Q | dO]
  // per buffer dS^T sits in front of P^T: with 64-query tiles the dQ MMA (M = 128) reads one 64-row atom past the
  // dS^T tile, which then falls inside the P^T tile of the same buffer (rows 64..127 of that product are never used)
  unsigned char *spds = sqdo + QS * C::kQStage;                   // [PB buffers][dS^T | P^T]
  unsigned char *sdq = spds + PB * C::kBufBytes;                  // [2][BQ rows of 128 bytes] dQ staging (1 KB aligned)
  unsigned char *sones = sdq + 2 * C::kDqStageBytes;             // the constant k-step of K and V
  unsigned char *sx = sones + C::kOnesBytes;                     // [QS stages][Q side | dO side] of that k-step
  uint64_t *bars = reinterpret_cast<uint64_t *>(sx + QS * 2 * C::kXBytes);
  uint64_t *kv_full = bars, *qdo_full = bars + 1, *qdo_empty = qdo_full + QS, *sdp_full = qdo_empty + QS, *sdp_read = sdp_full + 1;
  uint64_t *pds_full = sdp_read + 1, *dq_full = pds_full + 1, *dq_read = dq_full + 1;
  uint64_t *dkv_full = dq_read + 1, *pt_free = dkv_full + 1;
  uint64_t *dqs_written = pt_free + 1, *dqs_free = dqs_written + 1 /*[2]*/;
  uint64_t *x_full = dqs_free + 2 /*[QS]*/;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(x_full + QS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kb_lin = blockIdx.x;
  const int kb = kb_lin % a.kblocks_per_bucket;
  const int bj = (kb_lin / a.kblocks_per_bucket) % a.k;
  const int scope = kb_lin / (a.kblocks_per_bucket * a.k);
  const int head = blockIdx.y, brow = blockIdx.z;
  const uint32_t *my_scope = a.scopes + (size_t)scope * a.k;
  const int qtiles_per_bucket = a.bucket / BQ;
  const int num_qtiles = a.k * qtiles_per_bucket;
  const int key_tok = (int)my_scope[bj] * a.bucket + kb * kBK;

  if (threadIdx.x == 0) {
    tc::mbar_init(kv_full, 1);
    for (int s = 0; s < QS; ++s) { tc::mbar_init(&qdo_full[s], 1); tc::mbar_init(&qdo_empty[s], 1); }
    tc::mbar_init(sdp_full, 1); tc::mbar_init(sdp_read, 32 * C::kCW); tc::mbar_init(pds_full, 32 * C::kCW);
    tc::mbar_init(dq_full, 1); tc::mbar_init(dq_read, 32 * C::kCW); tc::mbar_init(dkv_full, 1);
    tc::mbar_init(dqs_written, 64 * (BQ < 128 ? BQ / 32 : 4)); tc::mbar_init(&dqs_free[0], 1); tc::mbar_init(&dqs_free[1], 1);
    tc::mbar_init(pt_free, 1);
    for (int s = 0; s < QS; ++s) tc::mbar_init(&x_full[s], 32);
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  // the constant k-step: every 16-byte half of every row is (1, 1, 1, 0, 0, 0, 0, 0), so that the product with a row
  // that carries its three terms in one half and zeros in the other does not depend on where the swizzle puts the
  // halves; the query-side rows start as zeros and only their first half is rewritten per tile
  for (int c = threadIdx.x; c < C::kOnesBytes / 16; c += C::kThreads)
    tc::sts128(tc::smem_u32(sones) + c * 16, make_uint4(0x3F803F80u, 0x00003F80u, 0u, 0u));
  for (int c = threadIdx.x; c < QS * 2 * C::kXBytes / 16; c += C::kThreads)
    tc::sts128(tc::smem_u32(sx) + c * 16, make_uint4(0u, 0u, 0u, 0u));
  tc::fence_proxy_async();
  if (warp == 1) { tc::tmem_alloc(tmem_slot, C::kTmemCols); tc::tmem_relinquish(); }
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_enter();
  tc::WaitCtx wc{abort_flag, a.status};

  if (warp == 0) {
    if (tc::elect_one()) {
      tc::tma_prefetch_desc(&map_q); tc::tma_prefetch_desc(&map_k); tc::tma_prefetch_desc(&map_v); tc::tma_prefetch_desc(&map_do);
      tc::mbar_expect_tx(kv_full, 2 * C::kKVBytes);
#pragma unroll
      for (int c = 0; c < C::NDCH; ++c) {
        tc::tma_load_3d(sk + c * kBK * C::RB, &map_k, kv_full, c * C::DCH, head, brow * a.L + key_tok);
        tc::tma_load_3d(sv + c * kBK * C::RB, &map_v, kv_full, c * C::DCH, head, brow * a.L + key_tok);
      }
      for (int i = 0; i < num_qtiles; ++i) {
        const int s = i % QS;
        const uint32_t ph = (uint32_t)(i / QS) & 1u;
        if (!tc::mbar_wait(&qdo_empty[s], ph ^ 1u, wc, 301, 200)) break;
        const int q_tok = (int)my_scope[i / qtiles_per_bucket] * a.bucket + (i % qtiles_per_bucket) * BQ;
        unsigned char *sq = sqdo + s * C::kQStage, *sdo = sq + C::kQBytes;
        tc::mbar_expect_tx(&qdo_full[s], C::kQStage);
#pragma unroll
        for (int c = 0; c < C::NDCH; ++c) {
          tc::tma_load_3d(sq + c * BQ * C::RB, &map_q, &qdo_full[s], c * C::DCH, head, brow * a.L + q_tok);
          tc::tma_load_3d(sdo + c * BQ * C::RB, &map_do, &qdo_full[s], c * C::DCH, head, brow * a.L + q_tok);
        }
      }
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc_s = tc::make_idesc_f16(kBK, BQ, true, false, false);          // S^T, dP^T
      constexpr uint32_t idesc_kv = tc::make_idesc_f16(kBK, C::DCH, true, false, true);      // dV, dK: B MN-major
      constexpr uint32_t idesc_dq = tc::make_idesc_f16(128, C::DCH, true, true, true);       // dQ: A and B MN-major
      // operand descriptors are a base and constant steps: built from addresses per product they cost the issuing thread,
      // which is on every tile's critical path, more than the products
      const uint64_t kd = tc::make_smem_desc(tc::smem_u32(sk), 16, 8 * C::RB, C::SWZ), vd = tc::make_smem_desc(tc::smem_u32(sv), 16, 8 * C::RB, C::SWZ);
      const uint64_t qd0 = tc::make_smem_desc(tc::smem_u32(sqdo), 16, 8 * C::RB, C::SWZ);
      const uint64_t onesd = tc::make_smem_desc(tc::smem_u32(sones), 16, 256, tc::kSwizzle32), xd0 = tc::make_smem_desc(tc::smem_u32(sx), 16, 256, tc::kSwizzle32);
      const uint64_t dsk0 = tc::make_smem_desc(tc::smem_u32(spds), 16, 1024, tc::kSwizzle128);            // dS^T (P^T) K-major
      const uint64_t dsm0 = tc::make_smem_desc(tc::smem_u32(spds), kBK * 128, 1024, tc::kSwizzle128);     // dS^T M-major
      // S^T = K Q^T and dP^T = V dO^T of the tile in ring stage s
      auto issue_s_dp = [&](int s) {
        const uint64_t qd = qd0 + (uint32_t)(s * (C::kQStage >> 4)), dod = qd + (uint32_t)(C::kQBytes >> 4), xd = xd0 + (uint32_t)(s * (2 * C::kXBytes >> 4));
#pragma unroll
        for (int c = 0; c < C::NDCH; ++c)
#pragma unroll
          for (int kk = 0; kk < C::DCH / 16; ++kk)
            tc::mma_f16_ss(tmem_base + C::kSCol, kd + (uint32_t)((c * kBK * C::RB >> 4) + 2 * kk), qd + (uint32_t)((c * BQ * C::RB >> 4) + 2 * kk), idesc_s, (c | kk) != 0);
        tc::mma_f16_ss(tmem_base + C::kSCol, onesd, xd, idesc_s, 1u);                       // - lse / scale
#pragma unroll
        for (int c = 0; c < C::NDCH; ++c)
#pragma unroll
          for (int kk = 0; kk < C::DCH / 16; ++kk)
            tc::mma_f16_ss(tmem_base + C::kDpCol, vd + (uint32_t)((c * kBK * C::RB >> 4) + 2 * kk), dod + (uint32_t)((c * BQ * C::RB >> 4) + 2 * kk), idesc_s, (c | kk) != 0);
        tc::mma_f16_ss(tmem_base + C::kDpCol, onesd, xd + (uint32_t)(C::kXBytes >> 4), idesc_s, 1u);      // - delta
        tc::mma_commit(sdp_full);
      };
      bool ok = tc::mbar_wait(kv_full, 0, wc, 302) && tc::mbar_wait(&qdo_full[0], 0, wc, 303) && tc::mbar_wait(&x_full[0], 0, wc, 315);
      if (ok) { tc::tc_fence_after_sync(); issue_s_dp(0); }
      int s = 0, ns = 1 % QS;                                     // ring stages of tile i and of tile i + 1
      uint32_t nph = QS == 1 ? 1u : 0u;
      for (int i = 0; i < num_qtiles && ok; ++i) {
        const int pb = i % PB;
        const bool more = i + 1 < num_qtiles;
        if (more && (!tc::mbar_wait(&qdo_full[ns], nph, wc, 303) || !tc::mbar_wait(&x_full[ns], nph, wc, 315))) { ok = false; break; }
        // every compute thread holds S^T and dP^T of tile i in registers: the next tile's scores are computed under this
        // tile's arithmetic
        if (!tc::mbar_wait(sdp_read, (uint32_t)i & 1u, wc, 316)) { ok = false; break; }
        tc::tc_fence_after_sync();
        if (more) issue_s_dp(ns);
        // P^T and dS^T of tile i are published
        if (!tc::mbar_wait(pds_full, (uint32_t)i & 1u, wc, 305)) { ok = false; break; }
        tc::tc_fence_after_sync();
        const uint64_t qd = qd0 + (uint32_t)(s * (C::kQStage >> 4)), dod = qd + (uint32_t)(C::kQBytes >> 4);
        const uint64_t dsk = dsk0 + (uint32_t)(pb * (C::kBufBytes >> 4)), ptk = dsk + (uint32_t)(C::kPBytes >> 4);
        // dV += P^T dO and dK += dS^T Q, 16 queries per instruction.  A = [keys x queries]: tensor memory (two bf16 per
        // column) when it fits, else shared-memory tiles with 128-byte rows of 64 queries
#pragma unroll
        for (int c = 0; c < C::NDCH; ++c) {
#pragma unroll
          for (int qk = 0; qk < BQ / 16; ++qk) {
            const uint32_t b_off = (uint32_t)(c * BQ * C::RB + qk * 16 * C::RB) >> 4, a_off = (uint32_t)((qk / 4) * (kBK * 128) + (qk % 4) * 32) >> 4;
            if (C::kTS) tc::mma_f16_ts(tmem_base + C::kDvCol + c * C::DCH, tmem_base + C::kPtCol + qk * 8, dod + b_off, idesc_kv, (i | qk) != 0);
            else tc::mma_f16_ss(tmem_base + C::kDvCol + c * C::DCH, ptk + a_off, dod + b_off, idesc_kv, (i | qk) != 0);
            tc::mma_f16_ss(tmem_base + C::kDkCol + c * C::DCH, dsk + a_off, qd + b_off, idesc_kv, (i | qk) != 0);
          }
        }
        tc::mma_commit(&qdo_empty[s]);
        if (C::kTS) tc::mma_commit(pt_free);
        // dQ_i = dS K_j: A = the dS^T tile read M-major (queries contiguous), K = keys in steps of 16 rows
        if (i > 0 && !tc::mbar_wait(dq_read, (uint32_t)(i - 1) & 1u, wc, 306)) { ok = false; break; }
        tc::tc_fence_after_sync();
        const uint64_t dsm = dsm0 + (uint32_t)(pb * (C::kBufBytes >> 4));
#pragma unroll
        for (int c = 0; c < C::NDCH; ++c)
#pragma unroll
          for (int ks = 0; ks < kBK / 16; ++ks)
            tc::mma_f16_ss(tmem_base + C::kDqCol + c * C::DCH, dsm + (uint32_t)(ks * 16 * 128 >> 4), kd + (uint32_t)((c * kBK * C::RB + ks * 16 * C::RB) >> 4), idesc_dq, ks != 0);
        tc::mma_commit(dq_full);
        if (i + 1 == num_qtiles) tc::mma_commit(dkv_full);
        s = ns;
        if (++ns == QS) { ns = 0; nph ^= 1u; }
      }
    }
  } else if (warp < 2 + C::kCW) {
    // Compute warps: kCW / 4 per tensor-memory lane quadrant; a thread owns one key row and, per query tile, the
    // BQ / 4 query columns of its warp.  After publishing tile i the warps read out dQ of tile i - 1 (queries on
    // the lanes) and add it to the fp32 scratch with vector reductions.
    const int cw = warp - 2;                          // 0..kCW-1
    const int q4 = warp & 3;                          // tensor-memory lane quadrant of this warp
    const int cidx = cw >> 2;                         // which part of the query columns
    const int ctid = cw * 32 + lane;                  // 0..32*kCW-1
    const int row = q4 * 32 + lane;                   // key row (S^T, dP^T, dK, dV) or query row (dQ)
    const uint32_t lane_off = (uint32_t)(q4 * 32) << 16;
    constexpr int QCOLS = C::QCOLS;                   // query columns per compute thread (32 or 16)
    constexpr int CH = C::kChunk;                     // of which one tensor-memory load brings in
    const int col0 = cidx * QCOLS;
    const uint64_t c2 = bpack2(a.scale_log2, a.scale_log2);
    bool ok = true;
    // dQ of tile i: two warps per quadrant take half of the D columns each
    auto read_out_dq = [&](int i) -> bool {
      if (!tc::mbar_wait(dq_full, (uint32_t)i & 1u, wc, 310)) return false;
      tc::tc_fence_after_sync();
      const int q_tok = (int)my_scope[i / qtiles_per_bucket] * a.bucket + (i % qtiles_per_bucket) * BQ;
      if constexpr (C::kTmaDq) {
        // The eight warps with cidx < 2 pull the tile out of tensor memory, release it, and write it to a staging
        // buffer in the 128-byte-swizzled layout of the scratch's tensor map; the drain warp hands the whole tile to
        // the copy engine as one add-reduce.  The compute warps issue no global reductions, so their next loads no
        // longer queue behind them (all sixteen warps sharing the read-out measured 1 % slower).
        // (with 64-query tiles the lanes of quadrants 2 and 3 hold no query: the dQ product has M = 128 rows)
        const bool stages = cidx < 2 && q4 * 32 < BQ;
        if (stages) {
          uint32_t o[16];
          tc::tmem_ld_32x32b_x16(tmem_base + lane_off + C::kDqCol + cidx * 16, o);
          const int buf = i & 1, use = i >> 1;
          // the add-reduce that last read this buffer (tile i - 2) has finished reading it
          if (use > 0 && !tc::mbar_wait(&dqs_free[buf], (uint32_t)(use - 1) & 1u, wc, 313)) return false;
          __syncwarp();
          const uint32_t stg = tc::smem_u32(sdq + buf * C::kDqStageBytes) + (uint32_t)row * 128u;
          tc::tmem_ld_wait();
          tc::tc_fence_before_sync();
          tc::mbar_arrive(dq_read);
#pragma unroll
          for (int h = 0; h < 4; ++h)
            tc::sts128(stg + (uint32_t)(((cidx * 4 + h) ^ (row & 7)) * 16), make_uint4(o[4 * h], o[4 * h + 1], o[4 * h + 2], o[4 * h + 3]));
          tc::fence_proxy_async();
          tc::mbar_arrive(dqs_written);
        } else {
          tc::mbar_arrive(dq_read);
        }
        return true;
      }
      if (cidx < 2) {
        float *dst = a.dq_acc + (((size_t)brow * a.L + q_tok + row) * a.H + head) * D + cidx * (D / 2);
        const bool live = row < BQ && q_tok + row < a.L;
#pragma unroll
        for (int c = 0; c < D / 2; c += 8) {
          uint32_t o[8];
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                       : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3]), "=r"(o[4]), "=r"(o[5]), "=r"(o[6]), "=r"(o[7])
                       : "r"(tmem_base + lane_off + C::kDqCol + cidx * (D / 2) + c) : "memory");
          tc::tmem_ld_wait();
          if (live) {
            atomicAdd(reinterpret_cast<float4 *>(dst + c), make_float4(__uint_as_float(o[0]), __uint_as_float(o[1]), __uint_as_float(o[2]), __uint_as_float(o[3])));
            atomicAdd(reinterpret_cast<float4 *>(dst + c + 4), make_float4(__uint_as_float(o[4]), __uint_as_float(o[5]), __uint_as_float(o[6]), __uint_as_float(o[7])));
          }
        }
      }
      tc::tc_fence_before_sync();
      tc::mbar_arrive(dq_read);
      return true;
    };
    for (int i = 0; i < num_qtiles && ok; ++i) {
      const int pb = i % PB;
      if (!tc::mbar_wait(sdp_full, (uint32_t)i & 1u, wc, 307)) { ok = false; break; }
      // the MMAs that read this shared-memory buffer (tile i - PB) must have finished; with two buffers the read-out of that
      // tile's dQ, behind the same products, has seen it
      if (PB == 1 && i > 0 && !tc::mbar_wait(dq_full, (uint32_t)(i - 1) & 1u, wc, 309)) { ok = false; break; }
      tc::tc_fence_after_sync();
      const uint32_t sds = tc::smem_u32(spds + pb * C::kBufBytes), spt = sds + C::kPBytes;
      const uint32_t prow = spt + (col0 / 64) * (kBK * 128) + row * 128;
      const uint32_t drow = sds + (col0 / 64) * (kBK * 128) + row * 128;
      // CH of the thread's QCOLS columns at a time (all of them, or 16 where two CTAs share the register file)
#pragma unroll
      for (int h0 = 0; h0 < QCOLS; h0 += CH) {
        const int colh = col0 + h0;
        uint32_t sr[CH], dr[CH];
        if (CH == 32) {
          tc::tmem_ld_32x32b_x32(tmem_base + lane_off + C::kSCol + colh, reinterpret_cast<uint32_t (&)[32]>(sr));
          tc::tmem_ld_32x32b_x32(tmem_base + lane_off + C::kDpCol + colh, reinterpret_cast<uint32_t (&)[32]>(dr));
        } else {
          tc::tmem_ld_32x32b_x16(tmem_base + lane_off + C::kSCol + colh, reinterpret_cast<uint32_t (&)[16]>(sr));
          tc::tmem_ld_32x32b_x16(tmem_base + lane_off + C::kDpCol + colh, reinterpret_cast<uint32_t (&)[16]>(dr));
        }
        tc::tmem_ld_wait();
        if (h0 + CH == QCOLS) {
          tc::tc_fence_before_sync();
          tc::mbar_arrive(sdp_read);
        }
        if (C::kTS && i > 0 && h0 == 0) {
          // the previous tile's dV / dK MMAs must have consumed the tensor-memory copies of P^T and dS^T
          if (!tc::mbar_wait(pt_free, (uint32_t)(i - 1) & 1u, wc, 313)) { ok = false; break; }
          tc::tc_fence_after_sync();
        }
#pragma unroll
        for (int v8 = 0; v8 < CH / 8; ++v8) {
          uint4 pw, dw;
          uint32_t *pw32 = reinterpret_cast<uint32_t *>(&pw), *dw32 = reinterpret_cast<uint32_t *>(&dw);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // the products hold s - lse / scale and dp - delta: p = 2^(c s'), ds = p dp', two queries per instruction
            float x0, x1;
            const uint64_t s2v = bpack2(__uint_as_float(sr[v8 * 8 + 2 * e]), __uint_as_float(sr[v8 * 8 + 2 * e + 1]));
            const uint64_t d2v = bpack2(__uint_as_float(dr[v8 * 8 + 2 * e]), __uint_as_float(dr[v8 * 8 + 2 * e + 1]));
            bunpack2(bmul2(s2v, c2), x0, x1);
            const float p0 = bwd_exp2(x0), p1 = bwd_exp2(x1);
            float g0, g1;
            bunpack2(bmul2(bpack2(p0, p1), d2v), g0, g1);
            const __nv_bfloat162 ph = __floats2bfloat162_rn(p0, p1), gh = __floats2bfloat162_rn(g0, g1);
            pw32[e] = *reinterpret_cast<const uint32_t *>(&ph);
            dw32[e] = *reinterpret_cast<const uint32_t *>(&gh);
          }
          const int chunk16 = ((colh % 64) / 8 + v8) ^ (row & 7);
          tc::sts128(drow + chunk16 * 16, dw);
          if (C::kTS) {
            tc::tmem_st_32x32b_x4(tmem_base + lane_off + C::kPtCol + colh / 2 + v8 * 4, pw.x, pw.y, pw.z, pw.w);
          } else {
            tc::sts128(prow + chunk16 * 16, pw);
          }
        }
      }
      if (!ok) break;
      if (C::kTS) tc::tmem_st_wait();
      tc::fence_proxy_async();
      tc::tc_fence_before_sync();
      tc::mbar_arrive(pds_full);
      if (i > 0 && !read_out_dq(i - 1)) { ok = false; break; }
    }
    if (ok) ok = read_out_dq(num_qtiles - 1);
    if (ok && tc::mbar_wait(dkv_full, 0, wc, 311) && cidx < 2 && key_tok + row < a.L) {
      tc::tc_fence_after_sync();
      const int wg = cidx;
      const size_t base = (((size_t)brow * a.L + key_tok + row) * a.H + head) * D + wg * (D / 2);
#pragma unroll
      for (int c = 0; c < D / 2; c += 8) {
        uint32_t kk[8], vv[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(kk[0]), "=r"(kk[1]), "=r"(kk[2]), "=r"(kk[3]), "=r"(kk[4]), "=r"(kk[5]), "=r"(kk[6]), "=r"(kk[7])
                     : "r"(tmem_base + lane_off + C::kDkCol + wg * (D / 2) + c) : "memory");
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(vv[0]), "=r"(vv[1]), "=r"(vv[2]), "=r"(vv[3]), "=r"(vv[4]), "=r"(vv[5]), "=r"(vv[6]), "=r"(vv[7])
                     : "r"(tmem_base + lane_off + C::kDvCol + wg * (D / 2) + c) : "memory");
        tc::tmem_ld_wait();
        uint4 kw, vw;
        __nv_bfloat162 *k2 = reinterpret_cast<__nv_bfloat162 *>(&kw), *v2 = reinterpret_cast<__nv_bfloat162 *>(&vw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          k2[e] = __floats2bfloat162_rn(__uint_as_float(kk[2 * e]) * a.scale, __uint_as_float(kk[2 * e + 1]) * a.scale);
          v2[e] = __floats2bfloat162_rn(__uint_as_float(vv[2 * e]), __uint_as_float(vv[2 * e + 1]));
        }
        *reinterpret_cast<uint4 *>(a.dK + base + c) = kw;
        *reinterpret_cast<uint4 *>(a.dV + base + c) = vw;
      }
    }
  } else if (warp == C::kConstWarp) {
    // Constants warp: -lse * sqrt(D) and -delta of every query tile as the rows of the extra k-step (three bf16 terms each,
    // exact to 2^-24), a stage ahead of the score products.  On the compute warps this cost the two that did it 450 cycles
    // of a tile's 2,200, and the others waited for them.
    constexpr int QL = (BQ + 31) / 32;                            // queries per lane
    auto split3 = [](float v, uint32_t &w0, uint32_t &w1) {
      const __nv_bfloat16 h0 = __float2bfloat16_rn(v);
      const float r1 = v - __bfloat162float(h0);
      const __nv_bfloat16 h1 = __float2bfloat16_rn(r1);
      const __nv_bfloat16 h2 = __float2bfloat16_rn(r1 - __bfloat162float(h1));
      w0 = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
      w1 = (uint32_t)__bfloat16_as_ushort(h2);
    };
    float l[QL], d[QL];
    auto fetch = [&](int i) {
      const int q_tok = (int)my_scope[i / qtiles_per_bucket] * a.bucket + (i % qtiles_per_bucket) * BQ;
#pragma unroll
      for (int q = 0; q < QL; ++q) {
        const size_t idx = ((size_t)brow * a.L + q_tok + q * 32 + lane) * a.H + head;
        l[q] = a.lse[idx];
        d[q] = a.delta[idx];
      }
    };
    fetch(0);
    for (int i = 0; i < num_qtiles; ++i) {
      const int s = i % QS;
      // the stage's last score products are behind the gradient products that free its Q and dO
      if (!tc::mbar_wait(&qdo_empty[s], ((uint32_t)(i / QS) & 1u) ^ 1u, wc, 317, 200)) break;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < QL; ++q) {
        const uint32_t base = tc::smem_u32(sx + s * 2 * C::kXBytes) + (uint32_t)(q * 32 + lane) * 32u;
        uint32_t w0, w1;
        split3(-l[q] * a.inv_scale, w0, w1);
        tc::sts128(base, make_uint4(w0, w1, 0u, 0u));
        split3(-d[q], w0, w1);
        tc::sts128(base + C::kXBytes, make_uint4(w0, w1, 0u, 0u));
      }
      tc::fence_proxy_async();
      tc::mbar_arrive(&x_full[s]);
      if (i + 1 < num_qtiles) fetch(i + 1);
    }
  } else if (C::kTmaDq && tc::elect_one()) {
    // Drain warp: one thread hands every staged dQ tile to the copy engine as an add-reduce into the fp32 scratch and
    // returns the staging buffer once the engine has read it, so no compute warp ever waits for the engine.
    bool ok = true;
    for (int i = 0; i < num_qtiles && ok; ++i) {
      const int buf = i & 1;
      if (!tc::mbar_wait(dqs_written, (uint32_t)i & 1u, wc, 314, 200)) { ok = false; break; }
      const int q_tok = (int)my_scope[i / qtiles_per_bucket] * a.bucket + (i % qtiles_per_bucket) * BQ;
      tc::tma_reduce_add_2d(&map_dq, sdq + buf * C::kDqStageBytes, head * D, brow * a.L + q_tok);
      tc::tma_commit();
      if (i > 0) {
        tc::tma_wait_read<1>();                         // the reduce of tile i - 1 has read its buffer
        tc::mbar_arrive(&dqs_free[buf ^ 1]);
      }
    }
    tc::tma_wait_all<0>();                              // every add-reduce of this CTA has landed
  }

  tc::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) { tc::tc_fence_after_sync(); tc::tmem_dealloc(tmem_base, C::kTmemCols); }
}

// Delta[b,t,h] = sum_d dO * O  (tests/test_attn_bwd.py:24-27)
__global__ void attn_bwd_delta_kernel(const __nv_bfloat16 *__restrict__ O, const __nv_bfloat16 *__restrict__ dO,
                                      float *__restrict__ delta, size_t rows, int D) {
  const uint32_t after = grid_enter();
  O += after; dO += after;
  size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const uint4 *po = reinterpret_cast<const uint4 *>(O + r * D), *pd = reinterpret_cast<const uint4 *>(dO + r * D);
  float acc = 0.f;
  for (int c = 0; c < D / 8; ++c) {
    uint4 a4 = __ldg(po + c), b4 = __ldg(pd + c);
    const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162 *>(&a4), *y = reinterpret_cast<const __nv_bfloat162 *>(&b4);
#pragma unroll
    for (int e = 0; e < 4; ++e) { float2 f = __bfloat1622float2(x[e]), g = __bfloat1622float2(y[e]); acc = fmaf(f.x, g.x, acc); acc = fmaf(f.y, g.y, acc); }
  }
  delta[r] = acc;
}

__global__ void attn_bwd_dq_convert_kernel(const float *__restrict__ acc, __nv_bfloat16 *__restrict__ dQ, size_t n8, float scale) {
  const uint32_t after = grid_enter();
  acc += after;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  float4 a4 = reinterpret_cast<const float4 *>(acc)[2 * i], b4 = reinterpret_cast<const float4 *>(acc)[2 * i + 1];
  uint4 w;
  __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&w);
  h[0] = __floats2bfloat162_rn(a4.x * scale, a4.y * scale); h[1] = __floats2bfloat162_rn(a4.z * scale, a4.w * scale);
  h[2] = __floats2bfloat162_rn(b4.x * scale, b4.y * scale); h[3] = __floats2bfloat162_rn(b4.z * scale, b4.w * scale);
  reinterpret_cast<uint4 *>(dQ)[i] = w;
}

// Clears the rows of the buckets that no scope lists in `mats` matrices of [batch][L rows of row16 16-byte words].  A block
// takes 32 buckets: it reads the whole table once (a few KB) and clears what is left over, which is nothing when the scopes
// cover every bucket.  (A zero fill of the gradients of an attention layer, 960,000 rows of 3 x 256, took 372 us.)
__global__ void __launch_bounds__(256) clear_unlisted_kernel(uint4 *__restrict__ t, const uint32_t *__restrict__ scopes, uint32_t entries,
                                                             uint32_t buckets, uint32_t bucket, uint32_t L, uint32_t row16, uint32_t mats) {
  const uint32_t after = grid_enter();
  scopes += after;
  __shared__ uint32_t listed;
  if (threadIdx.x == 0) listed = 0u;
  __syncthreads();
  const uint32_t b0 = blockIdx.x * 32;
  uint32_t mine = 0u;
  for (uint32_t e = threadIdx.x; e < entries; e += 256) {
    const uint32_t d = __ldg(scopes + e) - b0;
    if (d < 32u) mine |= 1u << d;
  }
  if (mine) atomicOr(&listed, mine);
  __syncthreads();
  const uint64_t words = (uint64_t)bucket * row16;                // of one bucket in one matrix
  for (uint32_t i = 0; i < 32 && b0 + i < buckets; ++i) {
    if ((listed >> i) & 1u) continue;
    for (uint32_t m = 0; m < mats; ++m) {
      uint4 *p = t + ((uint64_t)m * L + (uint64_t)(b0 + i) * bucket) * row16;
      for (uint64_t w = threadIdx.x; w < words; w += 256) p[w] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
}

template <int D>
static int launch_attn_bwd(const void *Q, const void *K, const void *V, const void *dO, AttnBwdArgs a, int device, cudaStream_t st) {
  using C = BwdCfg<D>;
  auto kern = attn_bwd_kernel<D>;
  F3D_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kern), device, C::kSmem));
  CUtensorMap mq, mk, mv, mdo;
  const uint64_t rows = (uint64_t)a.B * a.L;
  const uint64_t s1 = (uint64_t)D * 2, s2 = (uint64_t)a.H * D * 2;
  F3D_TRY(encode_tmap_3d(&mq, 0, Q, D, a.H, rows, s1, s2, C::DCH, 1, C::BQ, C::RB));
  F3D_TRY(encode_tmap_3d(&mdo, 0, dO, D, a.H, rows, s1, s2, C::DCH, 1, C::BQ, C::RB));
  F3D_TRY(encode_tmap_3d(&mk, 0, K, D, a.H, rows, s1, s2, C::DCH, 1, kBK, C::RB));
  F3D_TRY(encode_tmap_3d(&mv, 0, V, D, a.H, rows, s1, s2, C::DCH, 1, kBK, C::RB));
  // fp32 dQ scratch [B*L, H*D] as a tensor map for the add-reduce of a 128-row x 32-column tile (D = 32 only; the
  // other head sizes keep vector reductions and get a map they never use)
  CUtensorMap mdq = mq;
  if (C::kTmaDq)
    F3D_TRY(encode_tmap_2d(&mdq, 2, a.dq_acc, (uint64_t)a.H * D, rows, (uint64_t)a.H * D * 4, D, C::BQ, 128));
  dim3 grid(a.num_scopes * a.k * a.kblocks_per_bucket, a.H, a.B);
  launch(kern, grid, C::kThreads, C::kSmem, st, mq, mk, mv, mdo, mdq, a);
  return check_launch("buck_swin_bwd");
}

}  // namespace f3d

using namespace f3d;

extern "C" int f3d_buck_swin_bwd(const void *Q, const void *K, const void *V, const void *O, const void *dO, const void *LSE,
                                 void *Delta, void *dQ, void *dK, void *dV, const void *scope_buckets, int B, int L, int H,
                                 int D, int num_scopes, int scope_size, uint32_t bucket_size, int device, void *stream) {
  if (B <= 0 || L <= 0 || H <= 0) return set_error(F3D_ERR_ARG, "buck_swin_bwd: empty tensor");
  if (D != 16 && D != 32 && D != 64 && D != 128) return set_error(F3D_ERR_UNSUPPORTED, "buck_swin_bwd: head_dim %d (16, 32, 64, 128 are supported)", D);
  if (bucket_size == 0 || bucket_size % 128) return set_error(F3D_ERR_UNSUPPORTED, "buck_swin_bwd: bucket_size %u must be a positive multiple of 128", bucket_size);
  if (L % (int)bucket_size) return set_error(F3D_ERR_ARG, "buck_swin_bwd: sequence length %d is not a multiple of bucket_size %u", L, bucket_size);
  if (num_scopes < 0 || scope_size <= 0) return set_error(F3D_ERR_ARG, "buck_swin_bwd: Scope_buckets must be [S,k] with k > 0");
  if ((long long)H > 65535 || (long long)B > 65535) return set_error(F3D_ERR_UNSUPPORTED, "buck_swin_bwd: H and B must fit a grid dimension");
  DeviceGuard guard(device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  F3D_TRY(maybe_sync(st, "buck_swin_bwd"));
  const size_t rows = (size_t)B * L * H;
  launch(attn_bwd_delta_kernel, (unsigned)((rows + 255) / 256), 256, 0, st, static_cast<const __nv_bfloat16 *>(O), static_cast<const __nv_bfloat16 *>(dO),
                                                                       static_cast<float *>(Delta), rows, D);
  F3D_TRY(check_launch("buck_swin_bwd (delta)"));
  if (num_scopes == 0) {          // no bucket is listed: dQ is all zero, dK and dV have no listed rows
    F3D_CUDA_TRY(cudaMemsetAsync(dQ, 0, rows * D * sizeof(__nv_bfloat16), st));
    return maybe_sync(st, "buck_swin_bwd");
  }
  void *acc = nullptr;
  F3D_TRY(workspace(device, 2, rows * D * sizeof(float), st, &acc));
  F3D_CUDA_TRY(cudaMemsetAsync(acc, 0, rows * D * sizeof(float), st));
  const float scale = 1.f / sqrtf((float)D);
  AttnBwdArgs a{static_cast<const float *>(LSE), static_cast<const float *>(Delta), static_cast<float *>(acc),
                static_cast<__nv_bfloat16 *>(dK), static_cast<__nv_bfloat16 *>(dV), static_cast<const uint32_t *>(scope_buckets),
                B, L, H, num_scopes, scope_size, (int)bucket_size, (int)bucket_size / kBK, 1.4426950408889634f * scale, scale, sqrtf((float)D),
                status_word(device)};
  if (!a.status) return F3D_ERR_CUDA;
  int rc;
  switch (D) {
    case 16: rc = launch_attn_bwd<16>(Q, K, V, dO, a, device, st); break;
    case 32: rc = launch_attn_bwd<32>(Q, K, V, dO, a, device, st); break;
    case 64: rc = launch_attn_bwd<64>(Q, K, V, dO, a, device, st); break;
    default: rc = launch_attn_bwd<128>(Q, K, V, dO, a, device, st); break;
  }
  F3D_TRY(rc);
  const size_t n8 = rows * D / 8;
  launch(attn_bwd_dq_convert_kernel, (unsigned)((n8 + 255) / 256), 256, 0, st, static_cast<const float *>(acc), static_cast<__nv_bfloat16 *>(dQ), n8, scale);
  F3D_TRY(check_launch("buck_swin_bwd (dq convert)"));
  return maybe_sync(st, "buck_swin_bwd");
}

extern "C" int f3d_clear_unlisted(void *rows, const void *scope_buckets, int mats, int L, uint64_t row_bytes, int num_scopes,
                                  int scope_size, uint32_t bucket_size, int device, void *stream) {
  if (mats < 0 || L < 0 || num_scopes < 0 || scope_size < 0 || bucket_size == 0 || L % (int)bucket_size || row_bytes % 16 ||
      reinterpret_cast<uintptr_t>(rows) % 16)
    return set_error(F3D_ERR_ARG, "clear_unlisted: %d x %d rows of %llu bytes in buckets of %u", mats, L, (unsigned long long)row_bytes, bucket_size);
  const uint32_t buckets = (uint32_t)L / bucket_size;
  if (mats == 0 || buckets == 0 || row_bytes == 0) return F3D_OK;
  DeviceGuard guard(device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  launch(clear_unlisted_kernel, (buckets + 31) / 32, 256, 0, st, static_cast<uint4 *>(rows), static_cast<const uint32_t *>(scope_buckets),
                                                             (uint32_t)num_scopes * (uint32_t)scope_size, buckets, bucket_size, (uint32_t)L,
                                                             (uint32_t)(row_bytes / 16), (uint32_t)mats);
  F3D_TRY(check_launch("clear_unlisted"));
  return maybe_sync(st, "clear_unlisted");
}
