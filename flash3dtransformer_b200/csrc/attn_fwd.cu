// Bucketed (windowed) multi-head self-attention forward on tcgen05 tensor cores, sm_100a.
//
// Implements buck_swin_fwd(Q, K, V, O, L, Scope_buckets, bucket_size), which the reference's Python layer calls
// (flash3dxfmr/layers/buck_swin.py:57) but whose kernel source and binding are absent from the reference snapshot
// (declaration src/f3d_frontend.cu:90-92, binding commented out :136).  Semantics follow the reference's tests
// (tests/test_attn_fwd.py:295-452, tests/test_lib.py:24-48) and scope helpers (flash3dxfmr/psh/bucket_scope.py:
// 143-181): for every batch row b, head h and scope s (a row of Scope_buckets listing k buckets), the tokens of
// those buckets attend to each other with softmax(Q K^T / sqrt(D)) V; LSE is the natural-log row normaliser.
// Buckets that no scope lists are left untouched.
//
// Kernel shape: one CTA = 128 query rows of one (scope, head, batch row), 160 threads; four CTAs per SM up to D = 64, two
// at D = 128:
//   warp 0        one elected thread is both the TMA producer and the MMA issuer.  Keys come in tiles of 32 through a ring of
//                 four stages (3-D tensor maps over [token, head, dim], swizzle width = min(128, 2*D) bytes).  In turn i it
//                 waits for P of key tile i, issues O += P V (A operand P from tensor memory, V as MN-major B operand) and
//                 behind it S(i + 2) = Q K^T over the columns that P(i) occupies (products of one thread run in order), and
//                 commits both with one barrier.  A stage of the ring therefore holds V(i) and K(i + 2), and needs no barrier
//                 of its own to be refilled: P(i) comes from threads that have seen the commit of turn i - 2.
//   warps 1..4    softmax, one thread per query row: S is read with tcgen05.ld, P is written with tcgen05.st over the first
//                 half of the same columns; the epilogue normalises and stores O and LSE
// Two score buffers (2 x 32 columns) and O (D columns) share 128 tensor-memory columns (256 at D = 128).  With the scores of
// two tiles in flight the softmax threads hand over P and go on with the next tile without waiting for a product, one
// barrier wait per tile instead of two (the wait for S(j + 1) is also the wait for O to be complete up to tile j - 1), and
// D = 64 / 128 fit four / two CTAs on an SM where 64-key tiles with separate P columns fit two / one.
//
// What bounds it.  One exponential per score against 4*D tensor FLOPs: the special-function unit (16 per clock per SM) needs
// 512 cycles for 128 x 64 scores; three of every sixteen exponentials go to the FMA pipe (poly_exp2_pair), which leaves 416.
// The softmax loop alone, with every barrier satisfied and no products, takes 485 cycles there (four warps per scheduler),
// the kernel 550 including the start of its CTAs.  The loop takes no row maximum (SoftmaxRow::run): a 3-input maximum
// occupies the ALU and the FMA pipe together, and the scan was a tenth of the loop.
// Measured (B200, bf16, window 4096, TFLOP/s, before with 64-key tiles and one score buffer -> now): D = 16 248 -> 261,
// D = 32 490 -> 510, D = 64 626-662 -> 813-844, D = 128 737-790 -> 972.
// The issuing thread's code is on the critical path: unrolled by four it costs 8 % (instruction cache), as `lane == 0`
// instead of elect.sync 20 % (the compiler then serialises every uniform operand).
#include "f3d_common.cuh"
#include "tc_sm100.cuh"
#include "../../include/f3d_b200.h"

namespace f3d {

int *status_word(int device);

constexpr int kBQ = 128;      // query rows per tile
constexpr int kShortWindow = 8;     // query tiles of a scope up to which a CTA takes two (W = 1024)

// How query tiles map to CTAs: one each; two of a scope one after the other (kTwoTiles); one shared by several (kSplit).
// Builds of their own: the issuing thread's code is on the critical path, and what the plain mapping does not need costs it 2 %.
enum AttnMode : int { kPlain = 0, kTwoTiles = 1, kSplit = 2 };

struct AttnFwdArgs {
  __nv_bfloat16 *O; float *lse; const uint32_t *scopes;
  int B, L, H, num_scopes, k, bucket, q_blocks_per_bucket;   // q_blocks_per_bucket = bucket / 128
  float scale_log2;          // log2(e) / sqrt(D)
  int *status;
  int splits;                // kSplit: CTAs that share the keys of a query tile
  float *parts;              // kSplit without clusters: [query tile][part][D + 2][128] O, reference and sum of every part, and
  int *parts_done;           // [query tile] parts that have left theirs; zero before and after the launch
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

// packed fp32 pairs (Blackwell executes fma / add on two fp32 values per instruction)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// two fp32 values as a packed pair in the kernel's 16-bit element type (P in tensor memory, O in global memory)
template <bool F16> __device__ __forceinline__ uint32_t pack_p2(float a, float b) {
  if (F16) { __half2 h = __floats2half2_rn(a, b); return *reinterpret_cast<uint32_t *>(&h); }
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}

// 2^x for a pair of arguments (at most a few units above zero, any distance below) on the FMA pipe instead of the special-function unit: n = round(x) by the
// magic-number addition (the sum x + 1.5 * 2^23 carries n in its low mantissa bits), f = x - n in [-0.5, 0.5], a cubic
// for 2^f (largest relative error 7.5e-5, against the 3.9e-3 of the bf16 rounding P gets anyway), and n added to the
// exponent field with integer arithmetic.  The integer maximum keeps the result at 2^-126 or above (times the cubic),
// so arguments far below the range of an fp32 exponent come out as tiny numbers instead of wrapping around.
__device__ __forceinline__ void poly_exp2_pair(uint64_t x2, float &e0, float &e1) {
  const uint64_t magic2 = pack2(12582912.f, 12582912.f), nmagic2 = pack2(-12582912.f, -12582912.f);
  const uint64_t t2 = add2(x2, magic2);
  const uint64_t u2 = add2(t2, nmagic2);                              // n as a float, exact
  const uint64_t f2 = fma2(u2, pack2(-1.f, -1.f), x2);                // x - n
  uint64_t p2 = fma2(pack2(0.055171459913253784f, 0.055171459913253784f), f2, pack2(0.2426108568906784f, 0.2426108568906784f));
  p2 = fma2(p2, f2, pack2(0.6932609677314758f, 0.6932609677314758f));
  p2 = fma2(p2, f2, pack2(0.9999281167984009f, 0.9999281167984009f));
  float t0, t1, p0, p1;
  unpack2(t2, t0, t1);
  unpack2(p2, p0, p1);
  const int lowest = 0x4B400000 - 126;                                // bits of 1.5 * 2^23 - 126
  const int n0 = max(__float_as_int(t0), lowest), n1 = max(__float_as_int(t1), lowest);
  e0 = __int_as_float(__float_as_int(p0) + (n0 << 23));               // the bits of 1.5 * 2^23 vanish in the shift
  e1 = __int_as_float(__float_as_int(p1) + (n1 << 23));
}

template <int D> struct AttnCfg {
  static constexpr int BKV = 32;                    // keys per tile
  static constexpr int DCH = D < 64 ? D : 64;       // columns per swizzled row
  static constexpr int NDCH = D / DCH;
  static constexpr int RB = DCH * 2;                // bytes per swizzled row
  static constexpr uint64_t SWZ = RB == 128 ? tc::kSwizzle128 : (RB == 64 ? tc::kSwizzle64 : tc::kSwizzle32);
  static constexpr int kQBytes = kBQ * D * 2;
  static constexpr int kTileBytes = BKV * D * 2;    // one K or V tile
  static constexpr int R = 4;                       // ring stages: V of key tile i and K of key tile i + 2
  template <int MODE> static constexpr int q_bufs() { return MODE == kTwoTiles ? 2 : 1; }
  template <int MODE> static constexpr int smem() { return q_bufs<MODE>() * kQBytes + R * 2 * kTileBytes + 256 + 1024; }
  static constexpr int kThreads = 160;
  static constexpr uint32_t kOCol = 2 * BKV;        // S0 (P0 over its first 16 columns), S1, O
  static constexpr uint32_t kTmemCols = kOCol + D <= 128 ? 128 : 256;
  static constexpr int kMinCtas = 512 / kTmemCols;
  // parts of a split tile: 128 rows of O, reference and sum
  static_assert(kBQ * (D + 4) * 4 <= kQBytes + R * 2 * kTileBytes, "room for the parts of a split tile");
  // pairs of a tile whose exponentials go to the FMA pipe: every fifth, spread out so that both pipes work on every row
  // (an eighth to three eighths of the pairs measure within 2 % of one another)
  static constexpr int kPoly = 0x4210;
};

// One pair of scores: x = s * c - m on packed fp32 pairs, the exponentials on the special-function unit or (pairs in POLY)
// on the FMA pipe, the row sum of the unrounded probabilities, the packed 16-bit result.
template <int POLY, bool F16, bool GUARD>
__device__ __forceinline__ void exp_pair(const uint32_t (&r)[32], int i, uint64_t c2, uint64_t m2, uint64_t &sum2, uint32_t (&p)[16], float &poly_mx) {
  const uint64_t xx = fma2(pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), c2, m2);
  float e0, e1, x0, x1;
  unpack2(xx, x0, x1);
  if ((POLY >> i) & 1) {
    if (GUARD) poly_mx = max3(poly_mx, x0, x1);
    poly_exp2_pair(xx, e0, e1);
  } else {
    e0 = fast_exp2(x0); e1 = fast_exp2(x1);
  }
  sum2 = add2(sum2, pack2(e0, e1));
  p[i] = pack_p2<F16>(e0, e1);
}

__device__ __forceinline__ float row_max32(const uint32_t (&r)[32]) {
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int k = 0; k < 16; ++k) mx[k & 3] = max3(mx[k & 3], __uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
  return fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
}

__device__ __forceinline__ float sum4(uint64_t a, uint64_t b) {
  float s0, s1, s2, s3;
  unpack2(a, s0, s1);
  unpack2(b, s2, s3);
  return (s0 + s1) + (s2 + s3);
}

// Softmax state of one query row (one thread).
template <int D, bool F16> struct SoftmaxRow {
  using C = AttnCfg<D>;
  uint32_t tmem, tmem_o, s_full, p_full;            // scores and O in this warp's lanes; barrier addresses
  float m_run, l_run, alpha, poly_mx;
  uint64_t c2;
  bool ok, moved, bad;

  __device__ __forceinline__ void wait_s(int j, const tc::WaitCtx &wc) {
    ok = ok && tc::mbar_wait(s_full + 8u * ((uint32_t)j & 1u), (uint32_t)(j >> 1) & 1u, wc, 205);
    tc::tc_fence_after_sync();
  }
  __device__ __forceinline__ void rescale_o() {
#pragma unroll
    for (int c = 0; c < D; c += 16) {
      uint32_t o[16];
      tc::tmem_ld_32x32b_x16(tmem_o + c, o);
      tc::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
      tc::tmem_st_32x32b_x16(tmem_o + c, o);
    }
  }
  // key tile j, whose scores are in r: publishes P, fetches the scores of tile j + 1 into rn, returns the row sum.  The
  // wait for those scores is also the wait for O: their product was committed together with P V of tile j - 1.
  template <bool GUARD, bool FIRST>
  __device__ __forceinline__ float tile(int j, const uint32_t (&r)[32], uint32_t (&rn)[32], const tc::WaitCtx &wc) {
    const uint32_t b = (uint32_t)j & 1u;
    if (FIRST && moved) {
      wait_s(j + 1, wc);
      rescale_o();
    }
    const uint64_t m2 = pack2(-m_run, -m_run);
    uint64_t sa = pack2(0.f, 0.f), sb = sa;
    uint32_t p[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) exp_pair<C::kPoly, F16, GUARD>(r, i, c2, m2, (i & 1) ? sb : sa, p, poly_mx);
    wait_s(j + 1, wc);
    tc::tmem_ld_32x32b_x32(tmem + (b ^ 1u) * C::BKV, rn);
    tc::tmem_st_32x32b_x16(tmem + b * C::BKV, p);
    tc::tmem_ld_wait();
    tc::tmem_st_wait();
    tc::tc_fence_before_sync();
    tc::mbar_arrive(p_full + 8u * b);
    return sum4(sa, sb);
  }

  // The usual loop takes no maximum.  The reference m_run is the maximum of the first key tile; it moves by the exponent of
  // the row sum whenever that sum shows that scores have outgrown it, which leaves P, 16-bit floating point, and the fp32
  // sums as exact as any other reference.  What it cannot follow is a jump by more than 2^kJump within two tiles: such a
  // row marks itself bad and the CTA starts over with the maximum of every tile taken (`careful`).
  __device__ __forceinline__ void run(int j0, int n, uint32_t (&ra)[32], uint32_t (&rb)[32], float scale_log2, const tc::WaitCtx &wc) {
    constexpr float kMoveAt = 4096.f, kJump = F16 ? 16384.f : 1.2676506e30f;
    m_run = row_max32(ra) * scale_log2;
    for (int j = 0; j < n && ok; j += 2) {
      float s = tile<true, true>(j0 + j, ra, rb, wc);
      s += tile<true, false>(j0 + j + 1, rb, ra, wc);
      l_run += s;
      moved = __any_sync(0xFFFFFFFFu, !(s <= kMoveAt));
      if (moved) {
        bad = bad || !(s < kJump);
        const float up = s > kMoveAt ? (float)((__float_as_int(s) >> 23) - 127) : 0.f;
        alpha = fast_exp2(-up);
        m_run += up;
        l_run *= alpha;
      }
    }
    bad = bad || !(poly_mx < 100.f);
  }
  // The same with the maximum of every tile, for fp16 (whose P overflows past 65504) and for rows that `run` gave up on.
  // The reference still moves only when a maximum exceeds it by more than kMaxSlack (base-2 units), so that O is almost
  // never rescaled after the first tiles.
  __device__ __forceinline__ void run_careful(int j0, int n, uint32_t (&ra)[32], uint32_t (&rb)[32], float scale_log2, const tc::WaitCtx &wc) {
    for (int j = 0; j < n && ok; j += 2) {
      follow(row_max32(ra) * scale_log2, j > 0);
      l_run += tile<false, true>(j0 + j, ra, rb, wc);
      follow(row_max32(rb) * scale_log2, true);
      l_run += tile<false, true>(j0 + j + 1, rb, ra, wc);
    }
  }
  __device__ __forceinline__ void follow(float mx, bool have_o) {
    constexpr float kMaxSlack = 8.f;
    moved = __any_sync(0xFFFFFFFFu, mx > m_run + kMaxSlack);
    if (moved) {
      const float m_new = mx > m_run + kMaxSlack ? mx : m_run;
      alpha = fast_exp2(m_run - m_new);                                    // 1 for rows that keep their reference
      m_run = m_new;
      l_run *= alpha;
    }
    moved = moved && have_o;
  }
};

template <int D, bool F16, int MODE>
__global__ void __launch_bounds__(AttnCfg<D>::kThreads, AttnCfg<D>::kMinCtas)
attn_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, AttnFwdArgs a) {
  using C = AttnCfg<D>;
  constexpr int R = C::R, BKV = C::BKV;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *sq = smem, *sk = smem + C::template q_bufs<MODE>() * C::kQBytes, *sv = sk + R * C::kTileBytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(sv + R * C::kTileBytes);
  uint64_t *kv_full = bars, *s_full = bars + R, *p_full = s_full + 2, *q_full = p_full + 2 /*[2]*/;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(q_full + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_per_scope = a.k * a.q_blocks_per_bucket;
  constexpr bool SPLIT = MODE == kSplit;
  constexpr int nq = MODE == kTwoTiles ? 2 : 1;
  const int part = SPLIT ? blockIdx.x % a.splits : 0;            // the parts of a query tile are one cluster
  const int unit = SPLIT ? blockIdx.x / a.splits : blockIdx.x, units_per_scope = tiles_per_scope / nq;
  const int scope = unit / units_per_scope, qt = unit % units_per_scope * nq;
  const int head = blockIdx.y, brow = blockIdx.z;
  const uint32_t *my_scope = a.scopes + (size_t)scope * a.k;
// this CTA's keys: groups of 128 (always inside one bucket), [g0, g1) of the scope's; key tiles are a multiple of four
  const int g0 = SPLIT ? tiles_per_scope * part / a.splits : 0, g1 = SPLIT ? tiles_per_scope * (part + 1) / a.splits : tiles_per_scope;
  const int n = (g1 - g0) * (128 / BKV);
  const int slot0 = SPLIT ? g0 / a.q_blocks_per_bucket : 0, at0 = SPLIT ? (g0 % a.q_blocks_per_bucket) * 128 : 0;
  auto q_token = [&](int t) { return (int)my_scope[t / a.q_blocks_per_bucket] * a.bucket + (t % a.q_blocks_per_bucket) * kBQ; };
  const int row0 = brow * a.L;

  auto load_tile = [&](unsigned char *dst, const CUtensorMap *map, uint64_t *bar, int tok) {
#pragma unroll
    for (int c = 0; c < C::NDCH; ++c) tc::tma_load_3d(dst + c * BKV * C::RB, map, bar, c * C::DCH, head, tok);
  };
  uint32_t tmem_base = 0;
  tc::WaitCtx wc{abort_flag, a.status};
  SoftmaxRow<D, F16> sm;
  sm.ok = sm.bad = false;
  const int row = (warp & 3) * 32 + lane;                        // query row inside the tile = tensor-memory lane
  // normalised O and LSE of query tile qt + c
  auto store = [&](int c) {
    const int q_tok = q_token(qt + c);
    if (!sm.ok || q_tok + row >= a.L) return;
    const size_t tok = (size_t)row0 + q_tok + row;
    const float inv = 1.f / sm.l_run;
    __nv_bfloat16 *op = a.O + (tok * a.H + head) * D;
#pragma unroll
    for (int ch = 0; ch < D; ch += 16) {
      uint32_t o[16];
      tc::tmem_ld_32x32b_x16(sm.tmem_o + ch, o);
      tc::tmem_ld_wait();
      uint4 w[2];
      uint32_t *h2 = reinterpret_cast<uint32_t *>(w);
#pragma unroll
      for (int i = 0; i < 8; ++i) h2[i] = pack_p2<F16>(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
      *reinterpret_cast<uint4 *>(op + ch) = w[0];
      *reinterpret_cast<uint4 *>(op + ch + 8) = w[1];
    }
    a.lse[tok * a.H + head] = (sm.m_run + log2f(sm.l_run)) * 0.6931471805599453f;
  };
  for (int pass = 0; pass < 2; ++pass) {
    // One thread fills the ring and issues the products.  It sets the barriers up itself, so that its first loads are under
    // way before the CTA has its tensor memory.  Stage i of the ring holds V of key tile i and K of key tile i + 2; the first
    // four key tiles always lie in one bucket.
    if (warp == 0 && tc::elect_one()) {
      if (pass) for (uint64_t *bar = bars; bar <= q_full + 1; ++bar) tc::mbar_inval(bar);
      if (pass == 0) { tc::tma_prefetch_desc(&map_q); tc::tma_prefetch_desc(&map_k); tc::tma_prefetch_desc(&map_v); }
      *abort_flag = 0;
      for (int s = 0; s < R; ++s) tc::mbar_init(&kv_full[s], 1);
      for (int b = 0; b < 2; ++b) { tc::mbar_init(&s_full[b], 1); tc::mbar_init(&p_full[b], 128); }
      tc::mbar_init(&q_full[0], 1); tc::mbar_init(&q_full[1], 1);
      tc::mbar_fence_init();
      grid_wait();                                                // in the first pass; the kernel in front has long ended in the second
      const int q_tok = q_token(qt);
      const int tok0 = row0 + (int)my_scope[slot0] * a.bucket + at0;
      tc::mbar_expect_tx(q_full, C::kQBytes + 2 * C::kTileBytes);
#pragma unroll
      for (int c = 0; c < C::NDCH; ++c) tc::tma_load_3d(sq + c * kBQ * C::RB, &map_q, q_full, c * C::DCH, head, row0 + q_tok);
      for (int i = 0; i < 2; ++i) load_tile(sk + (R - 2 + i) * C::kTileBytes, &map_k, q_full, tok0 + i * BKV);
      for (int i = 0; i < 2; ++i) {
        tc::mbar_expect_tx(&kv_full[i], 2 * C::kTileBytes);
        load_tile(sv + i * C::kTileBytes, &map_v, &kv_full[i], tok0 + i * BKV);
        load_tile(sk + i * C::kTileBytes, &map_k, &kv_full[i], tok0 + (i + 2) * BKV);
      }
    }
    if (pass == 0 && warp == 1) { tc::tmem_alloc(tmem_slot, C::kTmemCols); tc::tmem_relinquish(); }
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    tmem_base = *tmem_slot;
    if (pass == 0) grid_enter();                                  // the other warps store O, which the kernel in front may still read
    if (warp == 0) {
      if (tc::elect_one()) {
        // position of a stream of key tiles: row inside its bucket, first token of the bucket and of the next one (the scope
        // table's entry is fetched a bucket ahead)
        struct Stream {
          const uint32_t *scope; int bucket, k, slot, row, base, next;
          __device__ __forceinline__ void init(const uint32_t *sc, int bk, int kk, int slot0, int from) {
            scope = sc; bucket = bk; k = kk; slot = slot0; row = from - BKV;
            base = (int)sc[slot] * bk;
            next = (int)sc[slot + 1 == kk ? 0 : slot + 1] * bk;
            take();
          }
          __device__ __forceinline__ int take() {
            const int t = base + row;
            row += BKV;
            if (row == bucket) {                                  // behind the last bucket the next query tile starts over
              row = 0;
              base = next;
              if (++slot == k) slot = 0;
              if (k > 1) next = (int)scope[slot + 1 == k ? 0 : slot + 1] * bucket;
            }
            return t;
          }
        } ks, vs;
        ks.init(my_scope, a.bucket, a.k, slot0, at0 + 4 * BKV);
        vs.init(my_scope, a.bucket, a.k, slot0, at0 + 2 * BKV);
        constexpr bool two = nq > 1;
        const int total = nq * n;
        auto load_stage = [&](int i) {
          const int s = i % R;
          const bool has_k = i + 2 < total;
          tc::mbar_expect_tx(&kv_full[s], has_k ? 2 * C::kTileBytes : C::kTileBytes);
          load_tile(sv + s * C::kTileBytes, &map_v, &kv_full[s], row0 + vs.take());
          if (has_k) load_tile(sk + s * C::kTileBytes, &map_k, &kv_full[s], row0 + ks.take());
        };
        constexpr uint32_t idesc_s = tc::make_idesc_f16(kBQ, BKV, !F16, false, false);
        constexpr uint32_t idesc_o = tc::make_idesc_f16(kBQ, C::DCH, !F16, false, true);       // B (= V) is MN-major
        const uint64_t qd = tc::make_smem_desc(tc::smem_u32(sq), 16, 8 * C::RB, C::SWZ);
        const uint64_t kd = tc::make_smem_desc(tc::smem_u32(sk), 16, 8 * C::RB, C::SWZ);
        const uint64_t vd = tc::make_smem_desc(tc::smem_u32(sv), 16, 8 * C::RB, C::SWZ);
        auto issue_s = [&](int slot, uint32_t b, bool second) {
          const uint64_t qds = two && second ? qd + (uint32_t)(C::kQBytes >> 4) : qd;
          const uint64_t kds = kd + (uint32_t)(slot * (C::kTileBytes >> 4));
#pragma unroll
          for (int c = 0; c < C::NDCH; ++c)
#pragma unroll
            for (int kk = 0; kk < C::DCH / 16; ++kk)
              tc::mma_f16_ss(tmem_base + b * BKV, qds + (uint32_t)(c * (kBQ * C::RB >> 4) + 2 * kk), kds + (uint32_t)(c * (BKV * C::RB >> 4) + 2 * kk),
                             idesc_s, (c | kk) != 0);
        };
        for (int i = 2; i < R - 2; ++i) load_stage(i);
        int rem = 0;                                              // key tile inside its query tile
        bool second = false;                                      // kTwoTiles: of the second query tile
        if (two) {
          tc::mbar_expect_tx(&q_full[1], C::kQBytes);
          tc::tma_load_3d(sq + C::kQBytes, &map_q, &q_full[1], 0, head, row0 + q_token(qt + 1));
        }
        bool ok = tc::mbar_wait(&q_full[0], 0, wc, 202);
        tc::tc_fence_after_sync();
        for (uint32_t b = 0; b < 2 && ok; ++b) {
          issue_s(R - 2 + b, b, false);
          tc::mma_commit(&s_full[b]);
        }
        for (int i = 0; i < total && ok; ++i) {
          const uint32_t b = (uint32_t)i & 1u;
          const int slot = i % R;
          // the two stages that carried K of tiles 0 and 1 have had no turn of their own yet
          if (!tc::mbar_wait(&kv_full[slot], (uint32_t)(i / R) & 1u, wc, 203)) { ok = false; break; }
          if (!tc::mbar_wait(&p_full[b], (uint32_t)(i >> 1) & 1u, wc, 204)) { ok = false; break; }
          tc::tc_fence_after_sync();
          const uint64_t vds = vd + (uint32_t)(slot * (C::kTileBytes >> 4));
#pragma unroll
          for (int c = 0; c < C::NDCH; ++c)
#pragma unroll
            for (int kk = 0; kk < BKV / 16; ++kk)                 // 16 keys per MMA: V rows kk * 16.., P columns kk * 8..
              tc::mma_f16_ts(tmem_base + C::kOCol + c * C::DCH, tmem_base + b * BKV + kk * 8,
                             vds + (uint32_t)(c * (BKV * C::RB >> 4) + kk * C::RB), idesc_o, ((two ? rem : i) | kk) != 0);
          // the next scores of this buffer overwrite P behind the product that reads it: MMAs of one thread run in order
          if (i + 2 < total) {
            if (two && rem + 2 == n) {
              second = true;
              if (!tc::mbar_wait(&q_full[1], 0u, wc, 202)) { ok = false; break; }
            }
            issue_s(slot, b, second);
          }
          tc::mma_commit(&s_full[b]);
          // P of tile i was written by threads that had seen the commit behind tile i - 2: its stage may be filled again
          if (i + R - 2 < total) load_stage(i + R - 2);
          if (two && ++rem == n) rem = 0;
        }
      }
    } else {
    sm.tmem = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);    // the tensor-memory lanes this warp may access
    sm.tmem_o = sm.tmem + C::kOCol;
    sm.s_full = tc::smem_u32(s_full);
    sm.p_full = tc::smem_u32(p_full);
    sm.c2 = pack2(a.scale_log2, a.scale_log2);
    sm.poly_mx = -INFINITY;
    sm.bad = false;
    sm.ok = true;
    uint32_t ra[32], rb[32];
    sm.wait_s(0, wc);
    tc::tmem_ld_32x32b_x32(sm.tmem, ra);
    tc::tmem_ld_wait();
    for (int c = 0; c < nq && sm.ok; ++c) {
      sm.m_run = -INFINITY;
      sm.l_run = 0.f;
      sm.alpha = 1.f;
      sm.moved = false;
      if (pass == 0) sm.run(c * n, n, ra, rb, a.scale_log2, wc);
      else sm.run_careful(c * n, n, ra, rb, a.scale_log2, wc);
      sm.wait_s((c + 1) * n + 1, wc);                             // behind the last product of this query tile
      if (pass == 0 && sm.moved) sm.rescale_o();                  // a reference that moved behind the last tile
      if (!SPLIT) store(c);
    }
    }
  if (pass == 1 || !__syncthreads_or(sm.ok && sm.bad)) break;
  }

  if (SPLIT && a.parts) {
    // The parts of a query tile meet in memory: each leaves its rows there, column by column, and the last one to do so adds
    // them up, in the order of the parts.
    __shared__ int last;
    const size_t tile = (size_t)(blockIdx.z * gridDim.y + blockIdx.y) * (gridDim.x / a.splits) + blockIdx.x / a.splits;
    float *const all = a.parts + tile * a.splits * kBQ * (D + 2) + row;                // this thread's row of every part
    constexpr int kPart = kBQ * (D + 2);
    if (warp != 0) {
      float *const mine = all + (size_t)part * kPart;
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        uint32_t o[16];
        tc::tmem_ld_32x32b_x16(sm.tmem_o + c, o);
        tc::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) mine[(c + i) * kBQ] = __uint_as_float(o[i]);
      }
      mine[D * kBQ] = sm.m_run;
      mine[(D + 1) * kBQ] = sm.l_run;
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.parts_done + tile, 1) == a.splits - 1;
    __syncthreads();
    const int q_tok = q_token(qt) + row;
    if (last && warp != 0 && q_tok < a.L) {
      __threadfence();
      float m = -INFINITY, l = 0.f;
      for (int p = 0; p < a.splits; ++p) m = fmaxf(m, __ldcg(all + (size_t)p * kPart + D * kBQ));
      for (int p = 0; p < a.splits; ++p)
        l = fmaf(fast_exp2(__ldcg(all + (size_t)p * kPart + D * kBQ) - m), __ldcg(all + (size_t)p * kPart + (D + 1) * kBQ), l);
      const float inv = 1.f / l;
      const size_t tok = (size_t)row0 + q_tok;
      __nv_bfloat16 *const out = a.O + (tok * a.H + head) * D;
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = 0.f;
        for (int p = 0; p < a.splits; ++p) {
          const float *o = all + (size_t)p * kPart;
          const float w = fast_exp2(__ldcg(o + D * kBQ) - m);
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = fmaf(w, __ldcg(o + (c + i) * kBQ), x[i]);
        }
#pragma unroll
        for (int i = 0; i < 16; i += 8)
          *reinterpret_cast<uint4 *>(out + c + i) = make_uint4(pack_p2<F16>(x[i] * inv, x[i + 1] * inv), pack_p2<F16>(x[i + 2] * inv, x[i + 3] * inv),
                                                               pack_p2<F16>(x[i + 4] * inv, x[i + 5] * inv), pack_p2<F16>(x[i + 6] * inv, x[i + 7] * inv));
      }
      a.lse[tok * a.H + head] = (m + log2f(l)) * 0.6931471805599453f;
    }
    if (last && threadIdx.x == 0) a.parts_done[tile] = 0;
  } else if (SPLIT) {
    // The parts of a query tile meet in shared memory: CTA p of the cluster receives every part's O, reference and sum of
    // `share` of the rows, over the operands nobody needs any more, and writes those rows.
    constexpr int kStride = D + 4;                                // floats per row of a part
    const int share = kBQ / a.splits;
    tc::cluster_sync();                                           // every CTA of the cluster is done with its operands
    if (warp != 0) {
      const int owner = row / share;
      const uint32_t dst = tc::mapa(tc::smem_u32(sq), owner) + (uint32_t)((part * share + row - owner * share) * kStride) * 4u;
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        uint32_t o[16];
        tc::tmem_ld_32x32b_x16(sm.tmem_o + c, o);
        tc::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) tc::sts_cluster128(dst + (uint32_t)(c + i) * 4u, make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]));
      }
      tc::sts_cluster128(dst + (uint32_t)D * 4u, make_uint4(__float_as_uint(sm.m_run), __float_as_uint(sm.l_run), 0u, 0u));
    }
    tc::cluster_sync();
    if (warp != 0 && sm.ok) {
      const float *parts = reinterpret_cast<const float *>(sq);
      const int step = share * kStride, q_tok = q_token(qt);
      for (int item = threadIdx.x - 32; item < share * (D / 8); item += 128) {
        const int r = item / (D / 8), ch = item % (D / 8) * 8, qr = part * share + r;
        if (q_tok + qr >= a.L) continue;
        const float *mine = parts + r * kStride;
        float m = -INFINITY, l = 0.f, x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int p = 0; p < a.splits; ++p) m = fmaxf(m, mine[p * step + D]);
        for (int p = 0; p < a.splits; ++p) {
          const float *o = mine + p * step;
          const float w = fast_exp2(o[D] - m);
          const float4 u = *reinterpret_cast<const float4 *>(o + ch), v = *reinterpret_cast<const float4 *>(o + ch + 4);
          l = fmaf(w, o[D + 1], l);
          x[0] = fmaf(w, u.x, x[0]); x[1] = fmaf(w, u.y, x[1]); x[2] = fmaf(w, u.z, x[2]); x[3] = fmaf(w, u.w, x[3]);
          x[4] = fmaf(w, v.x, x[4]); x[5] = fmaf(w, v.y, x[5]); x[6] = fmaf(w, v.z, x[6]); x[7] = fmaf(w, v.w, x[7]);
        }
        const float inv = 1.f / l;
        const size_t tok = (size_t)row0 + q_tok + qr;
        *reinterpret_cast<uint4 *>(a.O + (tok * a.H + head) * D + ch) =
            make_uint4(pack_p2<F16>(x[0] * inv, x[1] * inv), pack_p2<F16>(x[2] * inv, x[3] * inv), pack_p2<F16>(x[4] * inv, x[5] * inv),
                       pack_p2<F16>(x[6] * inv, x[7] * inv));
        if (ch == 0) a.lse[tok * a.H + head] = (m + log2f(l)) * 0.6931471805599453f;
      }
    }
  }

  tc::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) { tc::tc_fence_after_sync(); tc::tmem_dealloc(tmem_base, C::kTmemCols); }
}

template <int D, bool F16>
static int launch_attn_fwd(const void *Q, const void *K, const void *V, AttnFwdArgs a, int device, cudaStream_t st) {
  using C = AttnCfg<D>;
  const int dt = F16 ? 1 : 0;
  CUtensorMap mq, mk, mv;
  const uint64_t rows = (uint64_t)a.B * a.L;
  const uint64_t s1 = (uint64_t)D * 2, s2 = (uint64_t)a.H * D * 2;
  F3D_TRY(encode_tmap_3d(&mq, dt, Q, D, a.H, rows, s1, s2, C::DCH, 1, kBQ, C::RB));
  F3D_TRY(encode_tmap_3d(&mk, dt, K, D, a.H, rows, s1, s2, C::DCH, 1, C::BKV, C::RB));
  F3D_TRY(encode_tmap_3d(&mv, dt, V, D, a.H, rows, s1, s2, C::DCH, 1, C::BKV, C::RB));
  const int tiles_per_scope = a.k * a.q_blocks_per_bucket;
  const long long tiles = (long long)a.num_scopes * tiles_per_scope, heads = (long long)a.H * a.B;
  const long long room = (long long)sm_count(device) * C::kMinCtas;
  // A query tile is a chain of key tiles, 0.4 us each on an SM that has little else to do.  Where the tiles are so few that
  // the SMs would hold less than half of the CTAs they have room for, the keys of a tile are shared out to a cluster of two
  // or four CTAs (clusters of three, and five to eight, measure slower: they pack the SMs badly); a part keeps at least 512
  // keys, below which joining the parts costs what the split saves.  One head, D = 32, W = 4096: 12,288 tokens 49 -> 29 us
  // (four), 24,576 tokens 59 -> 45 us (two; four, which no longer fit at once: 48).
  a.splits = 1;
  while (a.splits < 4 && tiles * heads * a.splits * 2 <= room && tiles_per_scope / (2 * a.splits) >= 4) a.splits *= 2;
  // Where two CTAs a tile leave a third of the room empty and four do not fit at once, three do: packed into clusters they fit
  // badly, so they are launched by themselves and meet in memory (3-4 us more than a cluster needs).  One head, W = 4096:
  // 20,480 to 24,576 tokens D = 32 50 -> 39.5 us, 2 heads D = 64 57 -> 46.6; W = 2048: D = 32 28.8 -> 25.4; D = 128 46.4 -> 41.6.
  if (a.splits == 2 && tiles * heads * 3 <= room && tiles_per_scope / 3 >= 4) {
    void *parts = nullptr, *done = nullptr;
    if (workspace(device, 11, (size_t)(tiles * heads) * 3 * kBQ * (D + 2) * sizeof(float), st, &parts) == F3D_OK &&
        workspace(device, 12, (size_t)(tiles * heads) * sizeof(int), st, &done) == F3D_OK) {
      a.splits = 3;
      a.parts = static_cast<float *>(parts);
      a.parts_done = static_cast<int *>(done);
      auto kern = attn_fwd_kernel<D, F16, kSplit>;
      F3D_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kern), device, C::template smem<kSplit>()));
      launch(kern, dim3((unsigned)(tiles * 3), a.H, a.B), C::kThreads, C::template smem<kSplit>(), st, mq, mk, mv, a);
      return check_launch("buck_swin_fwd");
    }
    // (no scratch on a stream that captures before it ever ran this: the cluster of two)
  }
  if (a.splits > 1) {
    auto kern = attn_fwd_kernel<D, F16, kSplit>;
    F3D_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kern), device, C::template smem<kSplit>()));
    cudaLaunchAttribute cluster[2];
    cluster[0].id = cudaLaunchAttributeClusterDimension;
    cluster[0].val.clusterDim.x = (unsigned)a.splits;
    cluster[0].val.clusterDim.y = cluster[0].val.clusterDim.z = 1;
    cluster[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    cluster[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles * a.splits), a.H, a.B);
    cfg.blockDim = dim3(C::kThreads);
    cfg.dynamicSmemBytes = C::template smem<kSplit>();
    cfg.stream = st;
    cfg.attrs = cluster;
    cfg.numAttrs = 2;
    F3D_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, mq, mk, mv, a));
    return check_launch("buck_swin_fwd");
  }
  // A CTA spends 4,000 cycles before its first scores (tensor memory, scope table, Q and K from memory) and 1,300 after its
  // last: a fifth of its life at W = 512.  There it takes two query tiles of its scope, the second one's Q and keys arriving
  // under the first (8 heads: W = 512 1497 -> 1391 us, W = 1024 1253 -> 1202 us, W = 256 528 -> 495 us; four tiles: 1685, the
  // CTAs of an SM then run in step; nothing at W = 4096).
  if constexpr (D <= 32) {
    if (tiles_per_scope % 2 == 0 && tiles_per_scope <= kShortWindow && tiles * heads >= 8 * room) {
      auto kern = attn_fwd_kernel<D, F16, kTwoTiles>;
      F3D_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kern), device, C::template smem<kTwoTiles>()));
      launch(kern, dim3((unsigned)(tiles / 2), a.H, a.B), C::kThreads, C::template smem<kTwoTiles>(), st, mq, mk, mv, a);
      return check_launch("buck_swin_fwd");
    }
  }
  auto kern = attn_fwd_kernel<D, F16, kPlain>;
  F3D_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kern), device, C::template smem<kPlain>()));
  launch(kern, dim3((unsigned)tiles, a.H, a.B), C::kThreads, C::template smem<kPlain>(), st, mq, mk, mv, a);
  return check_launch("buck_swin_fwd");
}

template <bool F16>
static int launch_attn_fwd_any(int D, const void *Q, const void *K, const void *V, AttnFwdArgs a, int device, cudaStream_t st) {
  switch (D) {
    case 16: return launch_attn_fwd<16, F16>(Q, K, V, a, device, st);
    case 32: return launch_attn_fwd<32, F16>(Q, K, V, a, device, st);
    case 64: return launch_attn_fwd<64, F16>(Q, K, V, a, device, st);
    default: return launch_attn_fwd<128, F16>(Q, K, V, a, device, st);
  }
}

}  // namespace f3d

using namespace f3d;

static int buck_swin_fwd_impl(const void *Q, const void *K, const void *V, void *O, void *LSE, const void *scope_buckets,
                              int B, int L, int H, int D, int num_scopes, int scope_size, uint32_t bucket_size, int dtype,
                              int device, void *stream) {
  if (B <= 0 || L <= 0 || H <= 0) return set_error(F3D_ERR_ARG, "buck_swin_fwd: empty tensor");
  if (dtype != 0 && dtype != 1) return set_error(F3D_ERR_UNSUPPORTED, "buck_swin_fwd: element type %d (0 = bf16 and 1 = fp16 are supported)", dtype);
  if (D != 16 && D != 32 && D != 64 && D != 128) return set_error(F3D_ERR_UNSUPPORTED, "buck_swin_fwd: head_dim %d (16, 32, 64, 128 are supported)", D);
  if (bucket_size == 0 || bucket_size % kBQ) return set_error(F3D_ERR_UNSUPPORTED, "buck_swin_fwd: bucket_size %u must be a positive multiple of %d", bucket_size, kBQ);
  if (L % (int)bucket_size) return set_error(F3D_ERR_ARG, "buck_swin_fwd: sequence length %d is not a multiple of bucket_size %u", L, bucket_size);
  if (num_scopes < 0 || scope_size <= 0) return set_error(F3D_ERR_ARG, "buck_swin_fwd: Scope_buckets must be [S,k] with k > 0");
  if ((long long)H > 65535 || (long long)B > 65535) return set_error(F3D_ERR_UNSUPPORTED, "buck_swin_fwd: H and B must fit a grid dimension");
  if (num_scopes == 0) return F3D_OK;
  DeviceGuard guard(device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  F3D_TRY(maybe_sync(st, "buck_swin_fwd"));
  AttnFwdArgs a{static_cast<__nv_bfloat16 *>(O), static_cast<float *>(LSE), static_cast<const uint32_t *>(scope_buckets),
                B, L, H, num_scopes, scope_size, (int)bucket_size, (int)bucket_size / kBQ,
                1.4426950408889634f / sqrtf((float)D), status_word(device), 1};
  if (!a.status) return F3D_ERR_CUDA;
  F3D_TRY(dtype == 1 ? launch_attn_fwd_any<true>(D, Q, K, V, a, device, st) : launch_attn_fwd_any<false>(D, Q, K, V, a, device, st));
  return maybe_sync(st, "buck_swin_fwd");
}

extern "C" int f3d_buck_swin_fwd(const void *Q, const void *K, const void *V, void *O, void *LSE, const void *scope_buckets,
                                 int B, int L, int H, int D, int num_scopes, int scope_size, uint32_t bucket_size,
                                 int device, void *stream) {
  return buck_swin_fwd_impl(Q, K, V, O, LSE, scope_buckets, B, L, H, D, num_scopes, scope_size, bucket_size, 0, device, stream);
}

extern "C" int f3d_buck_swin_fwd_dtype(const void *Q, const void *K, const void *V, void *O, void *LSE, const void *scope_buckets,
                                       int B, int L, int H, int D, int num_scopes, int scope_size, uint32_t bucket_size,
                                       int dtype, int device, void *stream) {
  return buck_swin_fwd_impl(Q, K, V, O, LSE, scope_buckets, B, L, H, D, num_scopes, scope_size, bucket_size, dtype, device, stream);
}
