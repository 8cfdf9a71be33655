"""GPU parity of bucketed attention backward against autograd of the fp32 CPU oracle.

The reference accepts max < 4-8 and mean < 0.08-0.4 against FlashAttention's gradients
(tests/test_attn_bwd.py:176-376).  The bars here: for each of dQ, dK, dV the largest error is at most 2e-2 absolute
and at most 1 % of the tensor's largest entry, and the mean relative error exceeds the floor that rounding the exact
gradient to bf16 sets (1.42e-3) by at most 1.5e-3.  Measured on a B200 over every case of this file: largest error
5.5e-3 (0.62 % of the largest entry), mean relative error 2.2e-3 to 2.45e-3, i.e. 0.8e-3 to 1.04e-3 above the floor
(two bf16-rounded operands, P and dS, enter every product).  Every run appends its own figures to
gpurun_out/parity_achieved.jsonl.  Delta is compared with sum(dO * O) directly (tests/test_attn_bwd.py:24-27)."""
import pytest
import torch

from conftest import record_parity
from oracle import attn_oracle as ao

pytestmark = pytest.mark.gpu


def _run(dev, b, l, h, d, bucket, scopes, seed=0, mul=1.0):
    from flash3dtransformer_b200.lib import pshattn
    g = torch.Generator().manual_seed(seed)
    q, k, v, do = ((torch.randn(b, l, h, d, generator=g) * mul).bfloat16() for _ in range(4))
    sc = torch.tensor(scopes, dtype=torch.int64)
    scd = sc.to(torch.uint32).to(dev)
    qd, kd, vd, dod = (t.to(dev) for t in (q, k, v, do))
    o = torch.zeros_like(qd)
    lse = torch.zeros(b, l, h, device=dev)
    pshattn.buck_swin_fwd(qd, kd, vd, o, lse, scd, bucket)
    delta = torch.zeros(b, l, h, device=dev)
    dq, dk, dv = (torch.zeros_like(qd) for _ in range(3))
    pshattn.buck_swin_bwd(qd, kd, vd, o, dod, lse, delta, dq, dk, dv, scd, bucket)
    pshattn.device_status()
    rq, rk, rv, rdelta = ao.buck_swin_bwd(q, k, v, do, sc, bucket)
    exp_delta = (dod.float() * o.float()).sum(-1)
    return dict(dq=dq.float().cpu(), dk=dk.float().cpu(), dv=dv.float().cpu(), delta=delta.cpu(),
                rq=rq, rk=rk, rv=rv, rdelta=rdelta, exp_delta=exp_delta.cpu())


def _check_grad(name, got, ref, max_frac=0.01, mean_excess=1.5e-3, max_abs=2e-2):
    assert torch.isfinite(got).all(), name
    err = (got - ref).abs()
    rel = (err.mean() / ref.abs().mean()).item()
    floor = ((ref.bfloat16().float() - ref).abs().mean() / ref.abs().mean()).item()
    record_parity("attn_bwd_" + name, max_abs_raw=err.max().item(), ref_abs_max=ref.abs().max().item(), mean_rel_raw=rel,
                  rounding_floor=floor, bound_max_frac=max_frac, bound_mean_rel_excess=mean_excess)
    assert err.max().item() <= max_frac * ref.abs().max().item(), f"{name}: max err {err.max().item()} vs max {ref.abs().max().item()}"
    assert err.max().item() <= max_abs, f"{name}: max err {err.max().item()}"
    assert rel <= floor + mean_excess, f"{name}: mean rel {rel} (floor {floor})"


def _check_all(r):
    assert torch.allclose(r["delta"], r["exp_delta"], atol=1e-3, rtol=1e-3)          # exact definition on the GPU's own O
    assert (r["delta"] - r["rdelta"]).abs().max().item() <= 0.05                      # and close to the fp32 oracle's
    _check_grad("dQ", r["dq"], r["rq"])
    _check_grad("dK", r["dk"], r["rk"])
    _check_grad("dV", r["dv"], r["rv"])


@pytest.mark.parametrize("d", [16, 32, 64, 128])
def test_single_bucket_scopes(cuda_device, d):
    _check_all(_run(cuda_device, 2, 1024, 2, d, 256, [[0], [1], [2], [3]]))


@pytest.mark.parametrize("b,l,h,d,bucket,k", [(1, 4096, 4, 32, 512, 8), (2, 2048, 8, 32, 512, 2), (1, 1536, 2, 64, 128, 3),
                                             (1, 1280, 2, 128, 256, 5), (2, 2048, 4, 16, 512, 4), (1, 1280, 2, 32, 256, 5),
                                             (1, 3072, 2, 32, 128, 12)])
def test_multi_bucket_scopes(cuda_device, b, l, h, d, bucket, k):
    nb = l // bucket
    scopes = [list(range(i, i + k)) for i in range(0, nb, k)]
    _check_all(_run(cuda_device, b, l, h, d, bucket, scopes, seed=1))


@pytest.mark.parametrize("b,l,h,d,bucket,k", [(2, 2048, 2, 32, 128, 4), (1, 1536, 3, 32, 128, 3), (1, 2048, 2, 16, 256, 2),
                                             (1, 1024, 2, 32, 128, 1), (2, 1024, 1, 16, 512, 1)])
def test_small_windows(cuda_device, b, l, h, d, bucket, k):
    """Windows of at most 512 tokens at D <= 32 take the kernel that keeps every dQ tile in tensor memory (one CTA per
    scope and head, no scratch): 1 to 4 tiles per scope, buckets listed out of order."""
    nb = l // bucket
    scopes = [list(reversed(range(i, i + k))) for i in range(0, nb, k)]
    _check_all(_run(cuda_device, b, l, h, d, bucket, scopes, seed=11))


def test_unlisted_buckets_and_permutation(cuda_device):
    r = _run(cuda_device, 1, 2048, 2, 32, 256, [[0, 5], [2, 7]], seed=4)
    _check_all(r)
    for bk in (1, 3, 4, 6):
        for key in ("dq", "dk", "dv"):
            assert torch.all(r[key][:, bk * 256:(bk + 1) * 256] == 0)
    a = _run(cuda_device, 1, 1024, 2, 32, 256, [[0, 1, 2, 3]], seed=5)
    b = _run(cuda_device, 1, 1024, 2, 32, 256, [[2, 0, 3, 1]], seed=5)
    for key in ("dk", "dv"):
        assert torch.allclose(a[key], b[key], atol=2e-2, rtol=2e-2)


def test_uniform_attention_dv(cuda_device):
    """Q = 0 makes attention uniform: dV is the column mean of dO over the scope (tests/test_attn_bwd.py:406-439)."""
    from flash3dtransformer_b200.lib import pshattn
    dev = cuda_device
    l, h, d, bucket = 512, 2, 32, 256
    g = torch.Generator().manual_seed(7)
    q = torch.zeros(1, l, h, d, dtype=torch.bfloat16, device=dev)
    k, v, do = (torch.randn(1, l, h, d, generator=g).bfloat16().to(dev) for _ in range(3))
    sc = torch.tensor([[0, 1]], dtype=torch.uint32, device=dev)
    o = torch.zeros_like(q); lse = torch.zeros(1, l, h, device=dev); delta = torch.zeros(1, l, h, device=dev)
    dq, dk, dv = (torch.zeros_like(q) for _ in range(3))
    pshattn.buck_swin_fwd(q, k, v, o, lse, sc, bucket)
    pshattn.buck_swin_bwd(q, k, v, o, do, lse, delta, dq, dk, dv, sc, bucket)
    exp = do.float().mean(dim=1, keepdim=True).expand_as(do)
    assert torch.allclose(dv.float(), exp, atol=2e-3, rtol=2e-2)
    assert dk.float().abs().max().item() <= 1e-6          # Q = 0 kills dK


@pytest.mark.parametrize("bucket,l", [(256, 2048), (512, 4096)])
def test_partial_scope_table_with_poisoned_outputs(cuda_device, bucket, l):
    """dQ is defined for every token whichever kernel runs (windows of 512 tokens keep dQ in tensor memory, windows of
    1024 go through the fp32 scratch): rows of buckets no scope lists come back as zero even when the caller's buffer
    held NaN; dK and dV are written for listed buckets only and keep the caller's zero fill elsewhere."""
    from flash3dtransformer_b200.lib import pshattn
    dev = cuda_device
    h, d = 2, 32
    g = torch.Generator().manual_seed(21)
    q, k, v, do = (torch.randn(1, l, h, d, generator=g).bfloat16() for _ in range(4))
    scopes = [[0, 5], [2, 7]]
    sc = torch.tensor(scopes, dtype=torch.int64)
    scd = sc.to(torch.uint32).to(dev)
    qd, kd, vd, dod = (t.to(dev) for t in (q, k, v, do))
    o = torch.zeros_like(qd); lse = torch.zeros(1, l, h, device=dev)
    pshattn.buck_swin_fwd(qd, kd, vd, o, lse, scd, bucket)
    delta = torch.full((1, l, h), float("nan"), device=dev)
    dq = torch.full_like(qd, float("nan"))
    dk, dv = torch.zeros_like(qd), torch.zeros_like(qd)
    pshattn.buck_swin_bwd(qd, kd, vd, o, dod, lse, delta, dq, dk, dv, scd, bucket)
    pshattn.device_status()
    rq, rk, rv, _ = ao.buck_swin_bwd(q, k, v, do, sc, bucket)
    assert torch.isfinite(dq.float()).all() and torch.isfinite(delta).all()
    for bk in (1, 3, 4, 6):
        rows = slice(bk * bucket, (bk + 1) * bucket)
        assert torch.all(dq[:, rows] == 0) and torch.all(dk[:, rows] == 0) and torch.all(dv[:, rows] == 0)
    _check_grad("dQ", dq.float().cpu(), rq)
    _check_grad("dK", dk.float().cpu(), rk)
    _check_grad("dV", dv.float().cpu(), rv)


@pytest.mark.parametrize("k", [1, 8])
def test_full_size_layer_sampled_scopes_and_properties(cuda_device, k):
    """The attention-layer configuration at its full size (8 x 120,000 points padded to 960,000 tokens + tail, 8 heads x
    32, bucket 512, scope of 1 and of 8 buckets), forward and backward.  The CPU oracle cannot run 10^6 tokens in a test,
    so (a) a sample of scopes is cut out and compared with the oracle at the usual bars, and (b) size-independent
    properties are checked on the whole tensors: Delta = sum(dO * O) everywhere, V = 1 gives O = 1 and dQ = dK = 0,
    buckets that no scope lists keep what they held, and the result does not depend on what other scopes hold."""
    from flash3dtransformer_b200.lib import pshattn
    dev = cuda_device
    bucket, h, d = 512, 8, 32
    nb = 1880                                            # 962,560 tokens: 8 x 120,000 points and the padded tail
    l = nb * bucket
    g = torch.Generator(dev).manual_seed(k)
    q, kk, v, do = (torch.randn(1, l, h, d, device=dev, generator=g).bfloat16() for _ in range(4))
    listed = (nb // k) * k - 2 * k                       # the last buckets are listed by no scope
    sc = torch.arange(listed, dtype=torch.int64).reshape(-1, k)
    scd = sc.to(torch.uint32).to(dev)
    o = torch.full_like(q, 7.0); lse = torch.full((1, l, h), 7.0, device=dev); delta = torch.zeros(1, l, h, device=dev)
    dq, dk, dv = (torch.full_like(q, 7.0) for _ in range(3))
    pshattn.buck_swin_fwd(q, kk, v, o, lse, scd, bucket)
    pshattn.buck_swin_bwd(q, kk, v, o, do, lse, delta, dq, dk, dv, scd, bucket)
    pshattn.device_status()
    n_listed = listed * bucket
    assert torch.isfinite(o.float()).all() and torch.isfinite(dq.float()).all()
    # unlisted buckets: O, LSE, dK, dV untouched, dQ cleared (the documented contract of the backward)
    assert torch.all(o[:, n_listed:] == 7.0) and torch.all(lse[:, n_listed:] == 7.0)
    assert torch.all(dk[:, n_listed:] == 7.0) and torch.all(dv[:, n_listed:] == 7.0) and torch.all(dq[:, n_listed:] == 0)
    exp_delta = (do[:, :n_listed].float() * o[:, :n_listed].float()).sum(-1)
    assert torch.allclose(delta[:, :n_listed], exp_delta, atol=1e-3, rtol=1e-3)
    # sampled scopes against the oracle (a scope's result depends on its own tokens only)
    for s in (0, sc.shape[0] // 3, sc.shape[0] - 1):
        t0, t1 = int(sc[s, 0]) * bucket, (int(sc[s, -1]) + 1) * bucket
        cut = [t[:, t0:t1].cpu() for t in (q, kk, v, do)]
        local = torch.arange(k, dtype=torch.int64).reshape(1, k)
        ro, rlse = ao.buck_swin_fwd(cut[0], cut[1], cut[2], local, bucket)
        rq, rk, rv, _ = ao.buck_swin_bwd(cut[0], cut[1], cut[2], cut[3], local, bucket)
        err = (o[:, t0:t1].float().cpu() - ro).abs()
        floor = ((ro.bfloat16().float() - ro).abs().mean() / ro.abs().mean()).item()
        assert err.max().item() <= 2e-2 and (err.mean() / ro.abs().mean()).item() <= floor + 1e-3
        assert (lse[:, t0:t1].cpu() - rlse).abs().max().item() <= 2e-3
        _check_grad("dQ", dq[:, t0:t1].float().cpu(), rq)
        _check_grad("dK", dk[:, t0:t1].float().cpu(), rk)
        _check_grad("dV", dv[:, t0:t1].float().cpu(), rv)
    # V = 1: every output row is a convex combination of ones; its gradient with respect to the scores vanishes
    ones = torch.ones_like(v)
    o1 = torch.empty_like(q); lse1 = torch.empty_like(lse)
    pshattn.buck_swin_fwd(q, kk, ones, o1, lse1, scd, bucket)
    assert (o1[:, :n_listed].float() - 1).abs().max().item() <= 1e-2
    assert torch.equal(lse1[:, :n_listed], lse[:, :n_listed])          # the normaliser does not depend on V
    dq1, dk1, dv1 = (torch.empty_like(q) for _ in range(3))
    pshattn.buck_swin_bwd(q, kk, ones, o1, do, lse1, delta, dq1, dk1, dv1, scd, bucket)
    # dP = dO 1^T is constant along a row and Delta = sum(dO * O) is within rounding of it: dS ~ 0
    scale = do.float().abs().mean().item()
    assert dq1[:, :n_listed].float().abs().max().item() <= 0.05 * scale * 8
    assert dk1[:, :n_listed].float().abs().max().item() <= 0.05 * scale * 8


@pytest.mark.parametrize("b,d,listed", [(1, 32, [[0, 2], [5, 39]]), (2, 16, [[1], [33]]), (1, 64, [])])
def test_layer_gradient_of_unlisted_buckets_is_zero(cuda_device, b, d, listed):
    """The layer's gradients start uninitialised: the rows of buckets that no scope lists are cleared, the listed ones are what
    a zero-filled buffer gives."""
    from flash3dtransformer_b200.layers.buck_swin import BuckSwinFwdFunction, BuckSwinPackedFunction
    dev = cuda_device
    h, bucket, n = 2, 128, 40
    l = n * bucket
    g = torch.Generator(dev).manual_seed(0)
    qkv = torch.randn(3, b * l, h * d, generator=g, device=dev).bfloat16()
    do = torch.randn(b, l, h, d, generator=g, device=dev).bfloat16()
    sc = torch.tensor(listed if listed else [[0]], dtype=torch.int64).to(torch.uint32).to(dev)
    sc = sc if listed else sc[:0]
    rows = torch.zeros(l, dtype=torch.bool)
    for bk in [x for s in listed for x in s]:
        rows[bk * bucket:(bk + 1) * bucket] = True
    torch.empty(64 << 20, device=dev).fill_(float("nan"))             # what the allocator hands out next is not zero
    x = qkv.clone().requires_grad_(True)
    BuckSwinPackedFunction.apply(x, (b, l, h, d), sc, bucket).backward(do)
    parts = [qkv[i].view(b, l, h, d).clone().requires_grad_(True) for i in range(3)]
    BuckSwinFwdFunction.apply(*parts, sc, bucket).backward(do)
    for i in range(3):
        got = x.grad[i].view(b, l, h, d)
        assert torch.isfinite(got.float()).all() and torch.equal(got, parts[i].grad)
        assert torch.all(got[:, ~rows.to(dev)] == 0) and (not listed or got[:, rows.to(dev)].abs().max() > 0)
