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
    for (int i = 0; i < 3; ++i) { stats[i] = at; at += up(rows * 8); }
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
  for (int i = 0; i < count; ++i) {
    const f3d_xfmr_block &b = blocks[i];
    void *dst = (count - 1 - i) % 2 == 0 ? out : static_cast<void *>(base + s.ping);
    const bool fold = b.qkv_colsum != nullptr;
    if (fold) {
      // both LayerNorms ride in the projections behind them, on the row sums of the projections in front of them
      if (!stats) {
        stats = base + s.stats[0];
        F3D_TRY(f3d_row_stats_bf16(cur, stats, rows, channels, device, stream));
      }
      F3D_TRY(f3d_linear_fused(cur, b.qkv_w, b.qkv_b, nullptr, qkv, m, 3 * c, c, 3, 0, 0, stats, b.qkv_colsum, b.norm_eps, nullptr, device, stream));
    } else {
      F3D_TRY(f3d_layernorm_bf16(cur, b.norm_w, b.norm_b, norm, rows, channels, b.norm_eps, 0, device, stream));
      F3D_TRY(f3d_linear_fused(norm, b.qkv_w, b.qkv_b, nullptr, qkv, m, 3 * c, c, 3, 0, 0, nullptr, nullptr, 0.f, nullptr, device, stream));
    }
    F3D_TRY(f3d_buck_swin_fwd(q, q + mat, q + 2 * mat, attn, lse, b.scopes, 1, m, b.heads, c / b.heads, b.num_scopes, b.scope_size,
                              (uint32_t)b.bucket, device, stream));
    void *mid_stats = fold ? base + s.stats[2] : nullptr;
    F3D_TRY(f3d_linear_fused(attn, b.proj_w, b.proj_b, cur, mid, m, c, c, 1, 0, 0, nullptr, nullptr, 0.f, mid_stats, device, stream));
    if (fold) {
      F3D_TRY(f3d_linear_fused(mid, b.fc1_w, b.fc1_b, nullptr, hid, m, 2 * b.hidden, c, 1, 2, 0, mid_stats, b.fc1_colsum, b.ln2_eps, nullptr, device, stream));
    } else {
      F3D_TRY(f3d_layernorm_bf16(mid, b.ln2_w, b.ln2_b, norm, rows, channels, b.ln2_eps, 0, device, stream));
      F3D_TRY(f3d_linear_fused(norm, b.fc1_w, b.fc1_b, nullptr, hid, m, 2 * b.hidden, c, 1, 2, 0, nullptr, nullptr, 0.f, nullptr, device, stream));
    }
    // row sums of the block's output only where the next block folds its LayerNorm in
    const bool next_folds = i + 1 < count && blocks[i + 1].qkv_colsum != nullptr;
    void *next_stats = next_folds ? base + s.stats[(i + 1) % 2] : nullptr;
    F3D_TRY(f3d_linear_fused(hid, b.fc2_w, b.fc2_b, mid, dst, m, c, b.hidden, 1, 0, 0, nullptr, nullptr, 0.f, next_stats, device, stream));
    stats = next_stats;
    cur = dst;
  }
  return F3D_OK;
}
