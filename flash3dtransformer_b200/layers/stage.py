"""Transformer block and stage (mirror of the reference's flash3dxfmr/layers/stage.py:21-197).

XFMR keeps the reference's dataflow x -> norm -> attention -> + x -> MLP(with its own LayerNorm) -> + (stage.py:
90-101); the two residual additions are fused into the epilogues of the output projection and of the MLP's second
GEMM.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import List

import torch
import torch.cuda.nvtx as nvtx
from torch import nn
from torch.autograd import Function
from torch.nn.modules import module as nn_module

from . import buck_swin, elem_wise
from . import functional as F3
from ..lib import _cabi, pshattn
from ..psh import bucket_scope
from ..psh import dev_context as f3ddev
from ..psh import swin_attn as sa


@dataclass(slots=True)
class XFMRSpecs:
    channels: int
    hid_channels: int
    num_heads: int
    qkv_bias: bool
    swin_plan: bucket_scope.SwinPlan
    norm_layer: callable


class XFMR(nn.Module):
    NVTX_SCOPE = "XFMR"

    def __init__(self, channels: int, hid_chann: int, num_heads: int, buck_size: int, qkv_bias: bool,
                 swin_plan: bucket_scope.SwinPlan, norm_layer: callable):
        super().__init__()
        self.set_chnn = channels
        self.swin_plan = swin_plan
        self.norm = norm_layer(channels)
        self.bwa = buck_swin.BucketSwinAttentionModule(channels, num_heads, buck_size, qkv_bias)
        self.mlp = elem_wise.MLP(channels, hid_chann)

    def forward(self, reduced_coord, reduced_feat, reduced_sep):
        """(coords, features [N, C], seps) -> features [N, C]; coords and seps are unused, as in the reference."""
        assert reduced_feat.dim() == 2, f"Expect input features have two axes [N, C], but got shape={reduced_feat.shape}"
        n, c = reduced_feat.shape
        assert c == self.set_chnn, f"Expect input feat_dim={self.set_chnn}, but got {c}"
        scope_bucks = self.swin_plan.gen_scopes_from_plan(n, reduced_feat.device)
        if f3ddev.get_nvtx():
            nvtx.range_push(self.NVTX_SCOPE)
        feat = reduced_feat if reduced_feat.dtype == torch.bfloat16 else reduced_feat.to(torch.bfloat16)
        params = self._trainable(feat)
        if params is not None:
            out = XfmrBlockFunction.apply(feat, self, scope_bucks, *params)
        elif self._can_fold(feat):
            out = self._forward_folded(feat, reduced_feat, scope_bucks, n, c)
        else:
            x = F3.apply_norm(self.norm, feat)
            mid = self.bwa(x.view(1, n, c), scope_bucks, residual=feat).view(n, c)
            out = self.mlp(mid, residual=mid)
        if f3ddev.get_nvtx():
            nvtx.range_pop()
        return out

    def _trainable(self, feat):
        """The block's parameters when autograd can take the block as one node (XfmrBlockFunction), else None."""
        if not BlockStack.ENABLED or not torch.is_grad_enabled() or not feat.is_cuda or f3ddev.get_nvtx() or nn_module._has_any_global_hook():
            return None
        n, c = feat.shape
        ps = _plain_block(self)
        if ps is None or n == 0 or any(ps[i] is None for i in (0, 1, 2, 4, 6, 7, 8, 10)):
            return None
        f = ps[10].shape[1]
        if ((c != 32 and c % 64) or c > 1024 or f % 64 or tuple(self.norm.normalized_shape) != (c,) or self.bwa.head_dim not in (16, 32, 64, 128)
                or ps[8].shape[0] != 2 * f or any(p is not None and (p.device != feat.device or p.dtype != torch.float32) for p in ps)):
            return None
        return ps

    # Narrowest block that takes the folded path.  Measured per block on 16 x 120k points (LayerNorm kernels + four
    # GEMMs against four fused GEMMs): C = 32 / 64 / 128 lose 57 / 32 / 9 us (their epilogues are bound by instruction
    # issue, and a LayerNorm kernel over narrow rows costs only 45 us), C = 256 / 512 gain 39 / 75 us.
    FOLD_MIN_CHANNELS = 256

    def _can_fold(self, feat) -> bool:
        """Inference on the GPU with an affine nn.LayerNorm in front of the attention and the SwiGLU MLP, on rows wide
        enough for the fold to pay: both LayerNorms fold into the projections that follow them."""
        norm = self.norm
        return (not torch.is_grad_enabled() and feat.is_cuda and feat.shape[1] % 8 == 0 and isinstance(norm, nn.LayerNorm)
                and norm.elementwise_affine and norm.bias is not None and tuple(norm.normalized_shape) == (feat.shape[1],)
                and self.mlp.mlp.activation == "swiglu" and self.FOLD_MIN_CHANNELS <= feat.shape[1] <= 2048)

    def _forward_folded(self, feat, given, scope_bucks, n, c):
        """LN -> QKV, attention, proj + residual, LN -> fc1 (SwiGLU), fc2 + residual as four GEMMs and the attention
        kernel: no LayerNorm kernel runs.  Each LayerNorm is applied in the epilogue of the projection behind it from the
        row sums that the projection in front of it accumulated; the sums of this block's output travel with the
        returned tensor to the next block, and only a block whose input came from elsewhere (embedding, pooling,
        unpooling) computes them with a pass of its own."""
        stats = getattr(given, "_f3d_row_stats", None)
        if stats is None or stats.shape[0] != n:
            stats = F3.row_stats(feat)
        bwa, m = self.bwa, self.mlp.mlp
        qkv = F3.linear_inference(feat, bwa.qkv.weight, bwa.qkv.bias, nsplit=3, ln=(self.norm.weight, self.norm.bias, self.norm.eps),
                                  ln_stats=stats)
        attn_out = buck_swin.BuckSwinPackedFunction.apply(qkv, (1, n, bwa.num_heads, bwa.head_dim), scope_bucks, bwa.attn.buck_size)
        mid, mid_stats = F3.linear_inference(attn_out.view(n, c), bwa.proj.weight, bwa.proj.bias, residual=feat, want_stats=True)
        h = F3.linear_inference(mid, m.fc1_weight, m.fc1_bias, epilogue=F3.pshattn.EPI_SWIGLU,
                                ln=(m.layer_norm_weight, m.layer_norm_bias, m.eps), ln_stats=mid_stats)
        out, out_stats = F3.linear_inference(h, m.fc2_weight, m.fc2_bias, residual=mid, want_stats=True)
        out._f3d_row_stats = out_stats
        return out


class BlockStack:
    """Runs a list of XFMR blocks through one native call (f3d_xfmr_stack_bf16) where nothing but their forward is asked
    for: no autograd, no NVTX ranges, no hooks, the layer types of this package.  `run` returns None otherwise and the
    caller goes block by block; both give the same bits.

    What the call needs (pointers to the 16-bit weights, the folded LayerNorms, the scope tables) is laid out once per
    number of rows and stays valid as long as the blocks hold the same modules and unmodified parameters."""

    MAX_SIGNATURES = 32
    ENABLED = True

    def __init__(self):
        self._key, self._plans, self._keep = None, {}, ()

    def __reduce__(self):          # copies and pickles of a model start without a plan
        return (BlockStack, ())

    @staticmethod
    def _state(blocks):
        """(identity and version of everything the plan is made from, parameters per block), or None if a block is not
        the plain one."""
        key, params = [], []
        for b in blocks:
            if type(b) is not XFMR or b._forward_hooks or b._forward_pre_hooks:
                return None, None
            ps = _plain_block(b)
            if ps is None:
                return None, None
            for p in ps:
                if p is None:
                    key.append(None)
                else:
                    key += (id(p), p._version, p.data_ptr())
            key += (id(b.swin_plan), b.norm.eps, b.mlp.mlp.eps, b.bwa.num_heads, b.bwa.attn.buck_size)
            params.append(ps)
        return key, params

    def _build(self, blocks, params, n, c, device):
        """The argument array of the native call for n rows, and what its pointers need kept alive; None where the blocks
        have to run one by one."""
        arr, keep = (_cabi.XfmrBlock * len(blocks))(), []
        hidden = heads = 0

        def ptr(t):
            keep.append(t)
            return t.data_ptr()

        for a, b, ps in zip(arr, blocks, params):
            nw, nb, qw, qb, ow, ob, lw, lb, w1, b1, w2, b2 = ps
            if (nw is None or nb is None or tuple(b.norm.normalized_shape) != (c,) or b.set_chnn != c or any(p is not None and p.device != device for p in ps)):
                return None
            fold = XFMR.FOLD_MIN_CHANNELS <= c <= 2048
            a.norm_w, a.norm_b, a.ln2_w, a.ln2_b = (ptr(F3._fp32_param(p)) for p in (nw, nb, lw, lb))
            if fold:
                w, col, bias = F3.folded_layernorm(qw, qb, nw, nb)
                a.qkv_w, a.qkv_colsum, a.qkv_b = ptr(w), ptr(col), ptr(bias)
                w, col, bias = F3.folded_layernorm(w1, b1, lw, lb)
                a.fc1_w, a.fc1_colsum, a.fc1_b = ptr(w), ptr(col), ptr(bias)
            else:
                a.qkv_w, a.fc1_w = ptr(F3.bf16_weight(qw)), ptr(F3.bf16_weight(w1))
                a.qkv_b = ptr(F3._fp32_bias(qb)) if qb is not None else None
                a.fc1_b = ptr(F3._fp32_bias(b1)) if b1 is not None else None
            a.proj_w, a.fc2_w = ptr(F3.bf16_weight(ow)), ptr(F3.bf16_weight(w2))
            a.proj_b = ptr(F3._fp32_bias(ob)) if ob is not None else None
            a.fc2_b = ptr(F3._fp32_bias(b2)) if b2 is not None else None
            scopes = b.swin_plan.gen_scopes_from_plan(n, device)
            a.scopes = ptr(scopes)
            a.norm_eps, a.ln2_eps = b.norm.eps, b.mlp.mlp.eps
            a.heads, a.hidden = b.bwa.num_heads, w2.shape[1]
            a.num_scopes, a.scope_size, a.bucket = scopes.shape[0], scopes.shape[1], b.bwa.attn.buck_size
            hidden, heads = max(hidden, a.hidden), max(heads, a.heads)
        return arr, int(_cabi.load().f3d_xfmr_stack_scratch(n, c, hidden)), heads, tuple(keep)

    def run(self, blocks, x):
        if (not self.ENABLED or not x.is_cuda or torch.is_grad_enabled() or x.dim() != 2 or x.shape[1] % 8 or x.shape[0] == 0 or not len(blocks)
                or f3ddev.get_nvtx() or nn_module._has_any_global_hook()):
            return None
        key, params = self._state(blocks)
        if key is None:
            return None
        n, c = x.shape
        if key != self._key or len(self._plans) >= self.MAX_SIGNATURES:
            self._key, self._plans = key, {}
        plans = self._plans
        sig = (n, c, x.device, XFMR.FOLD_MIN_CHANNELS)
        if sig not in plans:
            plans[sig] = self._build(blocks, params, n, c, x.device)
        plan = plans[sig]
        if plan is None:
            return None
        feat = (x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16)).contiguous()
        out = torch.empty_like(feat)
        lse = sa.lse_rows(1, n, plan[2], x.device)
        scratch = torch.empty(plan[1], dtype=torch.uint8, device=x.device)
        st = _cabi.load().f3d_xfmr_stack_bf16(plan[0], len(blocks), feat.data_ptr(), out.data_ptr(), lse.data_ptr(), scratch.data_ptr(),
                                              plan[1], n, c, x.get_device(), pshattn._stream(x.get_device()))
        _cabi.check(st, "xfmr_stack")
        return out


def _plain_block(b):
    """The parameters of a block whose forward is all there is to it (the layer types of this package, no hooks inside), else
    None."""
    m = b._modules
    norm, bwa, mlp = m["norm"], m["bwa"], m["mlp"]
    if type(norm) is not nn.LayerNorm or type(bwa) is not buck_swin.BucketSwinAttentionModule or type(mlp) is not elem_wise.MLP:
        return None
    qkv, proj, inner = bwa._modules["qkv"], bwa._modules["proj"], mlp._modules["mlp"]
    if type(inner) is not elem_wise.LayerNormMLP or inner.activation != "swiglu" or type(qkv) is not nn.Linear or type(proj) is not nn.Linear:
        return None
    for mod in (norm, bwa, bwa._modules["attn"], qkv, proj, mlp, inner):
        if mod._forward_hooks or mod._forward_pre_hooks or mod._backward_hooks or mod._backward_pre_hooks:
            return None
    n, q, o, i = norm._parameters, qkv._parameters, proj._parameters, inner._parameters
    return (n["weight"], n["bias"], q["weight"], q["bias"], o["weight"], o["bias"], i["layer_norm_weight"], i["layer_norm_bias"],
            i["fc1_weight"], i["fc1_bias"], i["fc2_weight"], i["fc2_bias"])


class XfmrBlockFunction(Function):
    """A whole block as one autograd node: forward and backward are one native call each (f3d_xfmr_block_fwd_bf16,
    f3d_xfmr_block_bwd_bf16).  The same kernels as layer by layer, except that the residual gradients are added in fp32 inside
    the LayerNorm gradients and the pre-activation of the MLP is never stored."""

    @staticmethod
    def forward(ctx, x, block, scopes, *params):
        nw, nb, qw, qb, ow, ob, lw, lb, w1, b1, w2, b2 = params
        xb = (x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16)).contiguous()
        n, c = xb.shape
        h, f, dev = block.bwa.num_heads, w2.shape[1], xb.device
        # n1, attn, mid, n2 | qkv | hid of one allocation: they live and die together
        buf = torch.empty(n * (7 * c + f), dtype=torch.bfloat16, device=dev)
        row = n * c
        n1, attn, mid, n2 = (buf[i * row:(i + 1) * row].view(n, c) for i in range(4))
        qkv, hid = buf[4 * row:7 * row].view(3, n, c), buf[7 * row:].view(n, f)
        lse = torch.empty(n, h, dtype=torch.float32, device=dev)
        out = torch.empty_like(xb)
        a, keep = XfmrBlockFunction._block(block, scopes, params)
        t = _cabi.XfmrSaved(xb.data_ptr(), n1.data_ptr(), qkv.data_ptr(), attn.data_ptr(), lse.data_ptr(), mid.data_ptr(), n2.data_ptr(),
                            hid.data_ptr(), out.data_ptr())
        st = _cabi.load().f3d_xfmr_block_fwd_bf16(a, t, n, c, x.get_device(), pshattn._stream(x.get_device()))
        _cabi.check(st, "xfmr_block_fwd")
        ctx.save_for_backward(xb, buf, lse, *params)
        ctx.cfg = (block, scopes)
        return out

    @staticmethod
    def _block(block, scopes, params):
        """The native description of the block, and the tensors its pointers need kept alive."""
        nw, nb, qw, qb, ow, ob, lw, lb, w1, b1, w2, b2 = params
        keep = [F3._fp32_param(nw), F3._fp32_param(nb), F3.bf16_weight(qw), F3._fp32_bias(qb), F3.bf16_weight(ow), F3._fp32_bias(ob),
                F3._fp32_param(lw), F3._fp32_param(lb), F3.bf16_weight(w1), F3._fp32_bias(b1), F3.bf16_weight(w2), F3._fp32_bias(b2)]
        a = _cabi.XfmrBlock(*[None if t is None else t.data_ptr() for t in keep], None, None, scopes.data_ptr(), block.norm.eps,
                            block.mlp.mlp.eps, block.bwa.num_heads, w2.shape[1], scopes.shape[0], scopes.shape[1], block.bwa.attn.buck_size)
        return a, keep

    @staticmethod
    def backward(ctx, g):
        xb, buf, lse, *params = ctx.saved_tensors
        block, scopes = ctx.cfg
        nw, nb, qw, qb, ow, ob, lw, lb, w1, b1, w2, b2 = params
        n, c = xb.shape
        h, f, dev = block.bwa.num_heads, w2.shape[1], xb.device
        g = (g if g.dtype == torch.bfloat16 else g.to(torch.bfloat16)).contiguous()
        row = n * c
        p0 = buf.data_ptr()
        t = _cabi.XfmrSaved(xb.data_ptr(), p0, p0 + 8 * row, p0 + 2 * row, lse.data_ptr(), p0 + 4 * row, p0 + 6 * row, p0 + 14 * row, None)
        a, keep = XfmrBlockFunction._block(block, scopes, params)
        wt = (F3.bf16_weight_t(qw, 3), F3.bf16_weight_t(ow), F3.bf16_weight_t(w1), F3.bf16_weight_t(w2))
        # g_mid | g_qkv | g_pre, then the fp32 parameter gradients in one buffer each
        gbuf = torch.empty(n * (4 * c + 2 * f), dtype=torch.bfloat16, device=dev)
        gx = torch.empty_like(xb)
        flat = torch.empty(sum(p.numel() for p in params if p is not None), dtype=torch.float32, device=dev)
        grads, at = [], 0
        for p in params:
            if p is None:
                grads.append(None)
            else:
                grads.append(flat[at:at + p.numel()].view(p.shape))
                at += p.numel()
        q0, f0 = gbuf.data_ptr(), flat.data_ptr()
        # weights past the native kernel's limit take a library product from the same gradients
        native = [F3.native_wgrad(w.shape[0] // s, w.shape[1]) for w, s in ((qw, 3), (ow, 1), (w1, 1), (w2, 1))]
        ptr = [None if t is None else t.data_ptr() for t in grads]
        for i, ok in zip((2, 4, 8, 10), native):
            if not ok:
                ptr[i] = ptr[i + 1] = None
        gr = _cabi.XfmrGrads(*[w.data_ptr() for w in wt], *ptr, gx.data_ptr(), q0 + 8 * row, q0, q0 + 2 * row,
                             int(getattr(scopes, "_f3d_partition_of", -1) == n))
        lib = _cabi.load()
        size = int(lib.f3d_xfmr_block_bwd_scratch(n, c, f, h))
        scratch = torch.empty(size, dtype=torch.uint8, device=dev)
        st = lib.f3d_xfmr_block_bwd_bf16(a, t, gr, g.data_ptr(), scratch.data_ptr(), size, n, c, g.get_device(), pshattn._stream(g.get_device()))
        _cabi.check(st, "xfmr_block_bwd")
        if not all(native):
            n1, attn, n2, hid = buf[:row].view(n, c), buf[row:2 * row].view(n, c), buf[3 * row:4 * row].view(n, c), buf[7 * row:].view(n, f)
            g_mid, g_qkv, g_pre = gbuf[:row].view(n, c), gbuf[row:4 * row].view(3, n, c), gbuf[4 * row:].view(n, 2 * f)
            if not native[0]:
                for i in range(3):
                    F3.param_grads_into(g_qkv[i], n1, grads[2][i * c:(i + 1) * c], None if qb is None else grads[3][i * c:(i + 1) * c])
            for ok, gg, xx, i in ((native[1], g_mid, attn, 4), (native[2], g_pre, n2, 8), (native[3], g, hid, 10)):
                if not ok:
                    F3.param_grads_into(gg, xx, grads[i], grads[i + 1])
        grads = [None if t is None else t.to(p.dtype) for t, p in zip(grads, params)]
        return (gx, None, None, *grads)


class Stage(nn.Module):
    """Encoder blocks -> middle submodule -> decoder blocks, all with the (coord, feat, sep) signature."""
    NVTX_SCOPE = "Stage"

    def __init__(self, encoder_specs: List[XFMRSpecs], buck_size: int, submodule: nn.Module,
                 decoder_specs: List[XFMRSpecs]):
        super().__init__()
        if submodule is None:
            raise ValueError("A submodule must be provided for a Stage.")

        def block(spec):
            return XFMR(spec.channels, spec.hid_channels, spec.num_heads, buck_size, spec.qkv_bias, spec.swin_plan,
                        spec.norm_layer)

        self.encoder_blocks = nn.ModuleList([block(s) for s in encoder_specs])
        self.middle = submodule
        self.decoder_blocks = nn.ModuleList([block(s) for s in decoder_specs])
        self._encoder_stack, self._decoder_stack = BlockStack(), BlockStack()

    @staticmethod
    def _run(stack, blocks, coord, x, sep):
        out = stack.run(blocks, x)
        if out is None:
            for blk in blocks:
                x = blk(coord, x, sep)
            out = x
        return out

    def forward(self, reduced_coord, reduced_feat, reduced_sep):
        if f3ddev.get_nvtx():
            nvtx.range_push(self.NVTX_SCOPE)
        x = self._run(self._encoder_stack, self.encoder_blocks, reduced_coord, reduced_feat, reduced_sep)
        x = self.middle(reduced_coord, x, reduced_sep)
        x = self._run(self._decoder_stack, self.decoder_blocks, reduced_coord, x, reduced_sep)
        if f3ddev.get_nvtx():
            nvtx.range_pop()
        return x
