"""Operator calls through the native host module and through ctypes: the same results, and for bad arguments the same errors."""
import pytest
import torch

from flash3dtransformer_b200.lib import _cabi, pshattn


def _through_ctypes(monkeypatch):
    monkeypatch.setattr(_cabi, "_host", _cabi._NoHost)


def test_module_is_built_and_declines_other_arguments():
    h = _cabi.host()
    assert h is not _cabi._NoHost
    x = torch.zeros(4, 8)
    assert h.linear(x, x, None, x, None, 1, 0) is None                    # no CPU path
    assert h.linear() is None and h.bbox(1, 2, 3) is None and h.scatter(*[x] * 17) is None
    with pytest.raises(RuntimeError, match="not on a CUDA device"):
        pshattn.linear_bf16(x, x, None, x)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_same_results_as_through_ctypes(cuda_device, monkeypatch, dtype):
    from flash3dtransformer_b200.psh import psh_main
    rows, c = 1024, 64
    x = torch.randn(rows, c, device=cuda_device).to(dtype)
    w = torch.randn(3 * c, c, device=cuda_device).to(dtype)
    b, res = torch.randn(3 * c, device=cuda_device), torch.randn(rows, c, device=cuda_device).to(dtype)
    scopes = torch.arange(4, dtype=torch.int64).reshape(2, 2).to(torch.uint32).to(cuda_device)
    coords = torch.randn(3000, 3, device=cuda_device).half()
    seps = torch.tensor([1000, 3000], dtype=torch.int64).to(torch.uint32).to(cuda_device)

    def run():
        qkv = torch.empty(3, rows, c, device=cuda_device, dtype=dtype)
        pshattn.linear_bf16(x, w, b, qkv, nsplit=3)
        q, k, v = (t.view(1, rows, 2, 32) for t in qkv)
        o, lse, out = torch.empty_like(q), torch.empty(1, rows, 2, device=cuda_device), torch.empty_like(x)
        pshattn.buck_swin_fwd(q, k, v, o, lse, scopes, 256)
        pshattn.linear_bf16(o.view(rows, c), w[:c].contiguous(), None, out, residual=res)
        sc, buf = psh_main.batch_bucket_scatter(coords, seps, 256, 3328, 2)
        return [qkv, o, lse, out, sc.view(torch.int16), buf.bucket_id, buf.bucket_offs, *psh_main.scatter_index(buf, seps, 3328)]

    a = run()
    _through_ctypes(monkeypatch)
    for s, t in zip(a, run()):
        assert torch.equal(s.cpu(), t.cpu())


@pytest.mark.gpu
def test_same_errors_as_through_ctypes(cuda_device, monkeypatch):
    z = lambda *s, **k: torch.zeros(*s, device=cuda_device, **{"dtype": torch.bfloat16, **k})
    u = z(1, 2).to(torch.uint32)
    calls = [lambda: pshattn.linear_bf16(z(8, 64), z(64, 32), None, z(8, 64)), lambda: pshattn.linear_bf16(z(8, 64), z(64, 64), z(64), z(8, 64)),
             lambda: pshattn.linear_bf16(z(8, 64).float(), z(64, 64), None, z(8, 64)), lambda: pshattn.linear_bf16(z(8, 60), z(64, 60), None, z(8, 64)),
             lambda: pshattn.linear_bf16(z(64, 8).t(), z(64, 64), None, z(8, 64)),
             lambda: pshattn.buck_swin_fwd(*[z(1, 512, 1, 32)] * 4, z(1, 512, 2).float(), u, 256),
             lambda: pshattn.buck_swin_fwd(*[z(1, 512, 1, 48)] * 4, z(1, 512, 1).float(), u, 256),
             lambda: pshattn.bbox_f16(z(8, 3), z(3), z(3))]
    texts = []
    for native in (True, False):
        if not native:
            _through_ctypes(monkeypatch)
        for call in calls:
            with pytest.raises(RuntimeError) as e:
                call()
            texts.append(str(e.value))
    assert texts[:len(calls)] == texts[len(calls):]
