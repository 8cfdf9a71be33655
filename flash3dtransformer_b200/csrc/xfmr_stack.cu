// A run of transformer blocks of one width (the encoder or decoder list of a stage) issued by one call: inference only.
//
// The blocks are the reference's XFMR (flash3dxfmr/layers/stage.py:90-101): x -> norm -> attention -> + x -> MLP with a
// LayerNorm of its own -> +.  The kernels are the ones the operator entry points launch; what this call saves is the host's
// work between them.  Issued operator by operator from Python a 20,000-point forward (217 launches) takes the host 7.0 ms
// against 3.3 ms of kernels: the launches are what bounds every batch below half a million points.  All intermediates of a
// block live in one scratch buffer of the caller, reused from block to block.
#include "f3d_common.cuh"
#include "../../include/f3d_b200.h"

namespace f3d {

int linear_folded(const void *A, const void *W, const void *bias, const void *residual, void *C, int M, int N, int K, int nsplit, int epilogue,
                  const void *ln_stats, int ln_parts, const void *ln_colsum, float ln_eps, void *stats_out, int *stats_parts, int device,
                  cudaStream_t st);

struct StackScratch {
  // Q, K, V and the attention output of a block; the MLP's hidden rows take their place once the output projection is done
  size_t qkv, attn, hidden, norm, mid, ping, stats[3], total;
  StackScratch(size_t rows, size_t c, size_t hid) {
    const auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t row = up(rows * c * 2);
    qkv = hidden = 0;
    attn = up(3 * rows * c * 2);
    size_t at = attn + row;
    if (up(rows * hid * 2) > at) at = up(rows * hid * 2);
    norm = at; at += row;
    mid = at; at += row;
    ping = at; at += row;
    // row sums of a projection come in one part per column tile (32 columns at the least): the projection behind it adds them
    for (int i = 0; i < 3; ++i) { stats[i] = at; at += up(rows * 8 * ((c + 31) / 32)); }
    total = at;
  }
};

}  // namespace f3d

using namespace f3d;

extern "C" uint64_t f3d_xfmr_stack_scratch(uint32_t rows, uint32_t channels, uint32_t hidden) {
  return StackScratch(rows, channels, hidden).total;
}

extern "C" int f3d_xfmr_stack_bf16(const f3d_xfmr_block *blocks, int count, const void *x, void *out, void *lse,
                                   void *scratch, uint64_t scratch_bytes, uint32_t rows, uint32_t channels, int device, void *stream) {
  if (count <= 0 || !blocks) return set_error(F3D_ERR_ARG, "xfmr_stack: no blocks");
  if (rows == 0 || rows > 0x7FFFFFFFu || channels == 0) return set_error(F3D_ERR_ARG, "xfmr_stack: empty input");
  uint32_t hidden = 0;
  for (int i = 0; i < count; ++i) {
    if (blocks[i].heads <= 0 || channels % (uint32_t)blocks[i].heads) return set_error(F3D_ERR_ARG, "xfmr_stack: %u channels in %d heads", channels, blocks[i].heads);
    if ((uint32_t)blocks[i].hidden > hidden) hidden = (uint32_t)blocks[i].hidden;
  }
  const StackScratch s(rows, channels, hidden);
  if (scratch_bytes < s.total) return set_error(F3D_ERR_ARG, "xfmr_stack: %llu bytes of scratch, %llu are needed", (unsigned long long)scratch_bytes, (unsigned long long)s.total);
  char *base = static_cast<char *>(scratch);
  void *qkv = base + s.qkv, *attn = base + s.attn, *hid = base + s.hidden, *norm = base + s.norm, *mid = base + s.mid;
  const int m = (int)rows, c = (int)channels;
  char *q = static_cast<char *>(qkv);
  const size_t mat = (size_t)rows * channels * 2;
  const void *cur = x;
  void *stats = nullptr;                                          // row sums of cur, once a block has left them
  int parts = 1, mid_parts = 1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  for (int i = 0; i < count; ++i) {
    const f3d_xfmr_block &b = blocks[i];
    void *dst = (count - 1 - i) % 2 == 0 ? out : static_cast<void *>(base + s.ping);
    const bool fold = b.qkv_colsum != nullptr;
    if (fold) {
      // both LayerNorms ride in the projections behind them, on the row sums of the projections in front of them
      if (!stats) {
        stats = base + s.stats[0];
        parts = 1;
        F3D_TRY(f3d_row_stats_bf16(cur, stats, rows, channels, device, stream));
      }
      F3D_TRY(linear_folded(cur, b.qkv_w, b.qkv_b, nullptr, qkv, m, 3 * c, c, 3, 0, stats, parts, b.qkv_colsum, b.norm_eps, nullptr, nullptr, device, st));
    } else {
      F3D_TRY(f3d_layernorm_bf16(cur, b.norm_w, b.norm_b, norm, rows, channels, b.norm_eps, 0, device, stream));
      F3D_TRY(f3d_linear_fused(norm, b.qkv_w, b.qkv_b, nullptr, qkv, m, 3 * c, c, 3, 0, 0, nullptr, nullptr, 0.f, nullptr, device, stream));
    }
    F3D_TRY(f3d_buck_swin_fwd(q, q + mat, q + 2 * mat, attn, lse, b.scopes, 1, m, b.heads, c / b.heads, b.num_scopes, b.scope_size,
                              (uint32_t)b.bucket, device, stream));
    void *mid_stats = fold ? base + s.stats[2] : nullptr;
    F3D_TRY(linear_folded(attn, b.proj_w, b.proj_b, cur, mid, m, c, c, 1, 0, nullptr, 1, nullptr, 0.f, mid_stats, &mid_parts, device, st));
    if (fold) {
      F3D_TRY(linear_folded(mid, b.fc1_w, b.fc1_b, nullptr, hid, m, 2 * b.hidden, c, 1, 2, mid_stats, mid_parts, b.fc1_colsum, b.ln2_eps, nullptr, nullptr, device, st));
    } else {
      F3D_TRY(f3d_layernorm_bf16(mid, b.ln2_w, b.ln2_b, norm, rows, channels, b.ln2_eps, 0, device, stream));
      F3D_TRY(f3d_linear_fused(norm, b.fc1_w, b.fc1_b, nullptr, hid, m, 2 * b.hidden, c, 1, 2, 0, nullptr, nullptr, 0.f, nullptr, device, stream));
    }
    // row sums of the block's output only where the next block folds its LayerNorm in
    const bool next_folds = i + 1 < count && blocks[i + 1].qkv_colsum != nullptr;
    void *next_stats = next_folds ? base + s.stats[(i + 1) % 2] : nullptr;
    F3D_TRY(linear_folded(hid, b.fc2_w, b.fc2_b, mid, dst, m, c, b.hidden, 1, 0, nullptr, 1, nullptr, 0.f, next_stats, &parts, device, st));
    stats = next_stats;
    cur = dst;
  }
  return F3D_OK;
}

// ------------------------------------------------------------------------------------------------------- training
// The same block with what its backward pass needs kept, and that backward pass: 7 and 20 or 21 launches issued by one call each.
// Operator by operator autograd needed 33 ms of host time for a micro-batch that the GPU works on for 34 ms; what falls away
// besides are the additions of the residual gradients (they ride in the LayerNorm gradients) and the pre-activation of the MLP
// (its gradient is taken inside the product that recomputes it).
extern "C" int f3d_xfmr_block_fwd_bf16(const f3d_xfmr_block *blk, const f3d_xfmr_saved *t, uint32_t rows, uint32_t channels, int device, void *stream) {
  if (!blk || !t || rows == 0 || rows > 0x7FFFFFFFu || channels == 0 || blk->heads <= 0 || channels % (uint32_t)blk->heads)
    return set_error(F3D_ERR_ARG, "xfmr_block_fwd: %u rows of %u channels", rows, channels);
  const f3d_xfmr_block &b = *blk;
  const int m = (int)rows, c = (int)channels;
  char *q = static_cast<char *>(t->qkv);
  const size_t mat = (size_t)rows * channels * 2;
  F3D_TRY(f3d_layernorm_bf16(t->x, b.norm_w, b.norm_b, t->n1, rows, channels, b.norm_eps, 0, device, stream));
  F3D_TRY(f3d_linear_fused(t->n1, b.qkv_w, b.qkv_b, nullptr, t->qkv, m, 3 * c, c, 3, 0, 0, nullptr, nullptr, 0.f, nullptr, device, stream));
  F3D_TRY(f3d_buck_swin_fwd(q, q + mat, q + 2 * mat, t->attn, t->lse, b.scopes, 1, m, b.heads, c / b.heads, b.num_scopes, b.scope_size,
                            (uint32_t)b.bucket, device, stream));
  F3D_TRY(f3d_linear_fused(t->attn, b.proj_w, b.proj_b, t->x, t->mid, m, c, c, 1, 0, 0, nullptr, nullptr, 0.f, nullptr, device, stream));
  F3D_TRY(f3d_layernorm_bf16(t->mid, b.ln2_w, b.ln2_b, t->n2, rows, channels, b.ln2_eps, 0, device, stream));
  F3D_TRY(f3d_linear_fused(t->n2, b.fc1_w, b.fc1_b, nullptr, t->hid, m, 2 * b.hidden, c, 1, 2, 0, nullptr, nullptr, 0.f, nullptr, device, stream));
  return f3d_linear_fused(t->hid, b.fc2_w, b.fc2_b, t->mid, t->out, m, c, b.hidden, 1, 0, 0, nullptr, nullptr, 0.f, nullptr, device, stream);
}

namespace f3d {
// Widest block whose gradient of the hidden rows is formed inside the SwiGLU gradient.  Its tiles are narrow (64 hidden columns),
// so A is read more often, while 8 hid bytes a row need not move: with one to four k-blocks that is a gain (gradient of the hidden
// rows and of [gate | up], separately -> together: C = 32 at 1,605,632 rows 381 -> 218 us, C = 128 at 401,408 400 -> 278, C = 256
// at 200,704 456 -> 450 and at 22,912 62 -> 56), with eight it is a loss (C = 512 at 100,352 rows 661 -> 792 us).
constexpr int kMlpBwdMaxChannels = 256;

// gradient of the hidden rows first, where it is needed; once the pre-activation's gradient exists the [rows, C] intermediates
// take its place
struct BlockBwdScratch {
  size_t g_hid, g_n2, g_attn, g_n1, delta, total;
  BlockBwdScratch(size_t rows, size_t c, size_t hid, size_t heads) {
    const auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t row = up(rows * c * 2), first = c > (size_t)kMlpBwdMaxChannels ? up(rows * hid * 2) : 0;
    g_hid = g_n2 = 0;
    g_attn = row;
    g_n1 = 2 * row;
    delta = first > 3 * row ? first : 3 * row;
    total = delta + up(rows * heads * 4);
  }
};
}  // namespace f3d

extern "C" uint64_t f3d_xfmr_block_bwd_scratch(uint32_t rows, uint32_t channels, uint32_t hidden, uint32_t heads) {
  return BlockBwdScratch(rows, channels, hidden, heads).total;
}

extern "C" int f3d_xfmr_block_bwd_bf16(const f3d_xfmr_block *blk, const f3d_xfmr_saved *t, const f3d_xfmr_grads *gr, const void *grad_out, void *scratch,
                                       uint64_t scratch_bytes, uint32_t rows, uint32_t channels, int device, void *stream) {
  if (!blk || !t || !gr || rows == 0 || rows > 0x7FFFFFFFu || channels == 0 || blk->heads <= 0 || channels % (uint32_t)blk->heads)
    return set_error(F3D_ERR_ARG, "xfmr_block_bwd: %u rows of %u channels", rows, channels);
  const f3d_xfmr_block &b = *blk;
  const BlockBwdScratch s(rows, channels, (size_t)b.hidden, (size_t)b.heads);
  if (scratch_bytes < s.total) return set_error(F3D_ERR_ARG, "xfmr_block_bwd: %llu bytes of scratch, %llu are needed", (unsigned long long)scratch_bytes, (unsigned long long)s.total);
  char *base = static_cast<char *>(scratch);
  void *g_hid = base + s.g_hid, *g_n2 = base + s.g_n2, *g_attn = base + s.g_attn, *g_n1 = base + s.g_n1, *delta = base + s.delta;
  const int m = (int)rows, c = (int)channels, hid = b.hidden;
  const size_t mat = (size_t)rows * channels * 2;
  char *q = static_cast<char *>(t->qkv), *gq = static_cast<char *>(gr->g_qkv);
  const auto gemm = [&](const void *a, const void *wt, void *out, int n, int k) {
    return f3d_linear_fused(a, wt, nullptr, nullptr, out, m, n, k, 1, 0, 0, nullptr, nullptr, 0.f, nullptr, device, stream);
  };
  // MLP: fc2 and SwiGLU, fc1, LayerNorm (+ the residual gradient)
  if (gr->fc2_w) F3D_TRY(f3d_linear_wgrad_bf16(grad_out, t->hid, gr->fc2_w, gr->fc2_b, m, c, hid, device, stream));
  if (c <= kMlpBwdMaxChannels) {
    F3D_TRY(f3d_mlp_swiglu_bwd_bf16(t->n2, b.fc1_w, b.fc1_b, grad_out, gr->fc2_wt, gr->g_pre, m, hid, c, device, stream));
  } else {
    F3D_TRY(gemm(grad_out, gr->fc2_wt, g_hid, hid, c));
    F3D_TRY(f3d_linear_swiglu_bwd_bf16(t->n2, b.fc1_w, b.fc1_b, g_hid, gr->g_pre, m, 2 * hid, c, device, stream));
  }
  F3D_TRY(gemm(gr->g_pre, gr->fc1_wt, g_n2, c, 2 * hid));
  if (gr->fc1_w) F3D_TRY(f3d_linear_wgrad_bf16(gr->g_pre, t->n2, gr->fc1_w, gr->fc1_b, m, 2 * hid, c, device, stream));
  F3D_TRY(f3d_layernorm_bwd_add_bf16(t->mid, g_n2, b.ln2_w, grad_out, gr->g_mid, gr->ln2_w, gr->ln2_b, rows, channels, b.ln2_eps, device, stream));
  // attention: output projection, attention, QKV projection, LayerNorm (+ the residual gradient)
  F3D_TRY(gemm(gr->g_mid, gr->proj_wt, g_attn, c, c));
  if (gr->proj_w) F3D_TRY(f3d_linear_wgrad_bf16(gr->g_mid, t->attn, gr->proj_w, gr->proj_b, m, c, c, device, stream));
  if (!gr->covered) F3D_TRY(f3d_clear_unlisted(gr->g_qkv, b.scopes, 3, m, (uint64_t)channels * 2, b.num_scopes, b.scope_size, (uint32_t)b.bucket, device, stream));
  F3D_TRY(f3d_buck_swin_bwd(q, q + mat, q + 2 * mat, t->attn, g_attn, t->lse, delta, gq, gq + mat, gq + 2 * mat, b.scopes, 1, m, b.heads, c / b.heads,
                            b.num_scopes, b.scope_size, (uint32_t)b.bucket, device, stream));
  F3D_TRY(f3d_linear_ksplit_bf16(gr->g_qkv, gr->qkv_wt, nullptr, nullptr, g_n1, m, c, c, 3, device, stream));
  if (gr->qkv_w) F3D_TRY(f3d_linear_wgrad_split_bf16(gq, t->n1, gr->qkv_w, gr->qkv_b, m, 3 * c, c, 3, device, stream));
  return f3d_layernorm_bwd_add_bf16(t->x, g_n1, b.norm_w, gr->g_mid, gr->grad_x, gr->norm_w, gr->norm_b, rows, channels, b.norm_eps, device, stream);
}
