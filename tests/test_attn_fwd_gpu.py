"""GPU parity of bucketed attention forward against the fp32 CPU oracle.  Tolerance on N(0,1) bf16 inputs:
max abs <= 2e-2 against the fp32 oracle; mean|err| / mean|ref| exceeds the floor set by rounding the exact result to
bf16 (about 1.4e-3) by at most 1e-3; LSE max abs <= 2e-2.  Shapes follow the reference's tests
(tests/test_attn_fwd.py:295-452): (B,L,H,D) = (3,1280,2,128)/bucket 256, (16,4096,4,16)/512, (8,1280,2,128)/256."""
import pytest
import torch

from conftest import record_parity
from oracle import attn_oracle as ao

pytestmark = pytest.mark.gpu


def _run(dev, b, l, h, d, bucket, scopes, mul=1.0, seed=0):
    from flash3dtransformer_b200.lib import pshattn
    g = torch.Generator().manual_seed(seed)
    q, k, v = ((torch.randn(b, l, h, d, generator=g) * mul).bfloat16() for _ in range(3))
    sc = torch.tensor(scopes, dtype=torch.int64)
    o = torch.zeros(b, l, h, d, dtype=torch.bfloat16, device=dev)
    lse = torch.zeros(b, l, h, dtype=torch.float32, device=dev)
    pshattn.buck_swin_fwd(q.to(dev), k.to(dev), v.to(dev), o, lse, sc.to(torch.uint32).to(dev), bucket)
    pshattn.device_status()
    ref_o, ref_lse = ao.buck_swin_fwd(q, k, v, sc, bucket)
    return o.float().cpu(), lse.cpu(), ref_o, ref_lse


def _check(o, lse, ref_o, ref_lse, max_abs=2e-2, mean_rel=1e-3):
    assert torch.isfinite(o).all() and torch.isfinite(lse).all()
    err = (o - ref_o).abs() / ref_o.abs().clamp(min=1.0)
    rel = ((o - ref_o).abs().mean() / ref_o.abs().mean()).item()
    floor = ((ref_o.bfloat16().float() - ref_o).abs().mean() / ref_o.abs().mean()).item()
    record_parity("attn_fwd", max_abs_raw=(o - ref_o).abs().max().item(), max_abs_scaled=err.max().item(), mean_rel_raw=rel,
                  rounding_floor=floor, lse_max_abs=(lse - ref_lse).abs().max().item(), ref_abs_max=ref_o.abs().max().item(),
                  bound_max_abs=max_abs, bound_mean_rel_excess=mean_rel)
    assert err.max().item() <= max_abs, f"O max abs {err.max().item()}"
    assert rel <= floor + mean_rel, f"O mean rel {rel} (bf16 rounding floor {floor})"
    assert (lse - ref_lse).abs().max().item() <= max_abs, f"LSE max abs {(lse - ref_lse).abs().max().item()}"


@pytest.mark.parametrize("d", [16, 32, 64, 128])
def test_single_bucket_scopes(cuda_device, d):
    # 4 buckets of 256 tokens, every bucket its own scope
    _check(*_run(cuda_device, 2, 1024, 2, d, 256, [[0], [1], [2], [3]]))


@pytest.mark.parametrize("b,l,h,d,bucket,k", [(3, 1280, 2, 128, 256, 5), (2, 4096, 4, 16, 512, 4), (1, 4096, 4, 32, 512, 8),
                                             (2, 2048, 8, 32, 512, 2), (1, 1536, 2, 64, 128, 3)])
def test_multi_bucket_scopes(cuda_device, b, l, h, d, bucket, k):
    nb = l // bucket
    scopes = [list(range(i, i + k)) for i in range(0, nb, k)]
    _check(*_run(cuda_device, b, l, h, d, bucket, scopes, seed=1))


def test_permuted_buckets_inside_scope_and_unlisted_buckets(cuda_device):
    """The result does not depend on the order of the buckets inside a scope (tests/test_attn_fwd.py:418-452);
    buckets that no scope lists keep the caller's O."""
    a = _run(cuda_device, 1, 2048, 2, 32, 256, [[0, 1, 2, 3], [4, 5, 6, 7]], seed=3)
    b = _run(cuda_device, 1, 2048, 2, 32, 256, [[3, 1, 0, 2], [6, 7, 5, 4]], seed=3)
    _check(*a)
    assert torch.allclose(a[0], b[0], atol=1e-2) and torch.allclose(a[1], b[1], atol=1e-3)
    o, lse, ref_o, ref_lse = _run(cuda_device, 1, 2048, 2, 32, 256, [[0, 5], [2, 7]], seed=4)
    _check(o, lse, ref_o, ref_lse)
    for bk in (1, 3, 4, 6):
        assert torch.all(o[:, bk * 256:(bk + 1) * 256] == 0) and torch.all(lse[:, bk * 256:(bk + 1) * 256] == 0)


@pytest.mark.parametrize("mul", [2.0, 4.0, 16.0])
def test_scaled_inputs(cuda_device, mul):
    """Inputs scaled as in the reference's tests (x2 .. x16): the softmax becomes nearly one-hot.  The reference
    accepts max < 0.3-0.6 and mean < 0.01-0.02 against SDPA (tests/test_attn_fwd.py:319-368); the same bounds are
    used here relative to the input scale."""
    o, lse, ref_o, ref_lse = _run(cuda_device, 1, 1024, 2, 32, 256, [[0, 1], [2, 3]], mul=mul, seed=5)
    assert torch.isfinite(o).all() and torch.isfinite(lse).all()
    assert (o - ref_o).abs().max().item() <= 0.3 * mul / 2
    assert (o - ref_o).abs().mean().item() <= 0.01 * mul / 2
    assert ((lse - ref_lse).abs() / ref_lse.abs().clamp(min=1)).max().item() <= 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [16, 32, 64, 128])
@pytest.mark.parametrize("steps,bucket", [("first", 256), ("middle", 256), ("last", 256), ("ramp", 256), ("middle", 1024), ("ramp", 2048)])
def test_growing_scores(cuda_device, d, dtype, steps, bucket):
    """Rows whose later keys outgrow the reference taken from the first ones: a jump in the first, a middle or the last pair
    of 32-key tiles (past what the loop without a row maximum can follow: the careful pass) and a ramp it follows by moving
    its reference; in the larger buckets the keys of a query tile are shared out to two and four CTAs."""
    from flash3dtransformer_b200.lib import pshattn
    dev = cuda_device
    l, h = 2 * bucket, 2
    g = torch.Generator().manual_seed(11)
    q, k, v = (torch.randn(1, l, h, d, generator=g).to(dtype) for _ in range(3))
    big = 60.0 if dtype == torch.bfloat16 else 12.0
    gain = torch.ones(bucket)
    if steps == "ramp":
        gain = torch.linspace(1.0, 8.0, bucket)
    else:
        at = {"first": 40, "middle": 140, "last": bucket - 3}[steps]
        gain[at] = big
    k = (k.float() * gain.repeat(l // bucket)[None, :, None, None]).to(dtype)
    sc = torch.arange(l // bucket, dtype=torch.int64).reshape(-1, 1)
    o = torch.zeros(1, l, h, d, dtype=dtype, device=dev)
    lse = torch.zeros(1, l, h, dtype=torch.float32, device=dev)
    pshattn.buck_swin_fwd(q.to(dev), k.to(dev), v.to(dev), o, lse, sc.to(torch.uint32).to(dev), bucket)
    pshattn.device_status()
    ref_o, ref_lse = ao.buck_swin_fwd(q, k, v, sc, bucket)
    assert torch.isfinite(o.float()).all() and torch.isfinite(lse).all()
    assert (o.float().cpu() - ref_o).abs().max().item() <= 3e-2
    assert ((lse.cpu() - ref_lse).abs() / ref_lse.abs().clamp(min=1)).max().item() <= 1e-4


@pytest.mark.parametrize("d,dtype", [(16, torch.bfloat16), (32, torch.bfloat16), (32, torch.float16)])
@pytest.mark.parametrize("bucket,k,jump", [(256, 1, False), (128, 2, False), (512, 2, False), (256, 1, True)])
def test_many_short_scopes(cuda_device, d, dtype, bucket, k, jump):
    """So many tiles of a short window that a CTA takes two query tiles of its scope: the buckets of a scope in any order, and
    rows of the second tile that send the CTA into the careful pass.  Checked on the first, a middle and the last scope."""
    from flash3dtransformer_b200.lib import pshattn
    dev = cuda_device
    w, h = bucket * k, 16
    n = 5120 * 128 // (h * w) + 1                                 # scopes: past eight CTAs for every slot of 148 SMs
    l = n * w
    g = torch.Generator(dev).manual_seed(3)
    q, kk, v = (torch.randn(1, l, h, d, generator=g, device=dev).to(dtype) for _ in range(3))
    if jump:
        kk[:, 60::w] *= 12.0
        q[:, 128::w] *= 4.0
    sc = torch.randperm(l // bucket, generator=torch.Generator().manual_seed(4)).reshape(n, k)
    o = torch.zeros(1, l, h, d, dtype=dtype, device=dev)
    lse = torch.zeros(1, l, h, dtype=torch.float32, device=dev)
    pshattn.buck_swin_fwd(q, kk, v, o, lse, sc.to(torch.uint32).to(dev), bucket)
    pshattn.device_status()
    for s in (0, n // 2, n - 1):
        rows = torch.cat([torch.arange(b * bucket, (b + 1) * bucket) for b in sc[s].tolist()])
        sub = [t[:, rows.to(dev)].cpu() for t in (q, kk, v, o, lse)]
        ref_o, ref_lse = ao.buck_swin_fwd(sub[0], sub[1], sub[2], torch.arange(k).reshape(1, k), bucket)
        assert (sub[3].float() - ref_o).abs().max().item() <= 3e-2
        assert (sub[4] - ref_lse).abs().max().item() <= 2e-2


@pytest.mark.parametrize("l,h,d,bucket,k,dtype", [(24576, 1, 32, 512, 8, torch.bfloat16), (9728, 2, 16, 256, 19, torch.bfloat16), (10240, 2, 64, 512, 4, torch.float16),
                                                  (12288, 1, 128, 512, 8, torch.bfloat16), (19968, 1, 32, 512, 3, torch.float16)])
@pytest.mark.parametrize("jump", [False, True])
def test_three_parts_of_a_tile(cuda_device, l, h, d, bucket, k, dtype, jump):
    """Tile counts that three CTAs a tile fill the GPU with: parts of unequal length, a row whose scores send one part into the
    careful pass, the same bits on a second run (the counters are back at zero).  Checked on the last scope."""
    from flash3dtransformer_b200.lib import pshattn
    dev = cuda_device
    g = torch.Generator(dev).manual_seed(5)
    q, kk, v = (torch.randn(1, l, h, d, generator=g, device=dev).to(dtype) for _ in range(3))
    if jump:
        kk[:, bucket * k - 5::bucket * k] *= 12.0
        q[:, 7::128] *= 4.0
    sc = torch.arange(l // bucket).reshape(-1, k)
    runs = []
    for _ in range(2):
        o = torch.zeros(1, l, h, d, dtype=dtype, device=dev)
        lse = torch.zeros(1, l, h, dtype=torch.float32, device=dev)
        pshattn.buck_swin_fwd(q, kk, v, o, lse, sc.to(torch.uint32).to(dev), bucket)
        runs.append((o, lse))
    pshattn.device_status()
    assert torch.equal(runs[0][0], runs[1][0]) and torch.equal(runs[0][1], runs[1][1])
    rows = slice(l - bucket * k, l)
    sub = [t[:, rows].cpu() for t in (q, kk, v, runs[0][0], runs[0][1])]
    ref_o, ref_lse = ao.buck_swin_fwd(sub[0], sub[1], sub[2], torch.arange(k).reshape(1, k), bucket)
    assert (sub[3].float() - ref_o).abs().max().item() <= 3e-2
    assert (sub[4] - ref_lse).abs().max().item() <= 2e-2


def test_errors(cuda_device):
    from flash3dtransformer_b200.lib import pshattn
    dev = cuda_device
    q = torch.zeros(1, 512, 2, 32, dtype=torch.bfloat16, device=dev)
    lse = torch.zeros(1, 512, 2, device=dev)
    sc = torch.zeros(1, 1, dtype=torch.uint32, device=dev)
    with pytest.raises(RuntimeError, match="multiple"):
        pshattn.buck_swin_fwd(q, q, q, q.clone(), lse, sc, 96)
    with pytest.raises(RuntimeError, match="head_dim"):
        q2 = torch.zeros(1, 512, 2, 24, dtype=torch.bfloat16, device=dev)
        pshattn.buck_swin_fwd(q2, q2, q2, q2.clone(), lse, sc, 256)
    with pytest.raises(RuntimeError, match="dtype"):
        pshattn.buck_swin_fwd(q.float(), q, q, q, lse, sc, 256)
    with pytest.raises(RuntimeError, match="four axes"):
        pshattn.buck_swin_fwd(q[0], q[0], q[0], q[0], lse, sc, 256)
