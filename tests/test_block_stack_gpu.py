"""The native call for a run of blocks gives the bits of the blocks run one by one, follows changes of the parameters and
the modules, and steps aside where the module tree is more than its forward (hooks, autograd)."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def _stage(dev, c, depth, head_dim=32):
    from flash3dtransformer_b200 import configs, layers
    torch.manual_seed(0)
    spec = configs.hourglass_specs([c], [depth], head_dim=head_dim)[0]
    return layers.Stage(spec.encoder_specs, 512, torch.nn.Identity(), spec.decoder_specs).to(dev)


class _Middle(torch.nn.Module):
    def forward(self, coord, feat, sep):
        return feat.clone()           # a tensor of its own, as pooling and unpooling return


def _both(stage, x):
    from flash3dtransformer_b200.layers import stage as st
    with torch.no_grad():
        a = stage(None, x, None)
        st.BlockStack.ENABLED = False
        try:
            b = stage(None, x, None)
        finally:
            st.BlockStack.ENABLED = True
    return a, b


@pytest.mark.parametrize("c,depth,rows", [(32, 1, 512), (32, 2, 4096), (64, 3, 4608), (256, 1, 4096), (256, 3, 1024), (512, 2, 8192)])
def test_same_bits_as_block_by_block(cuda_device, c, depth, rows):
    stage = _stage(cuda_device, c, depth)
    stage.middle = _Middle()
    x = torch.randn(rows, c, device=cuda_device).bfloat16()
    a, b = _both(stage, x)
    assert torch.isfinite(a.float()).all() and torch.equal(a, b)
    assert stage._encoder_stack._plans and not torch.equal(a, x)


def test_follows_parameters_modules_and_hooks(cuda_device):
    stage = _stage(cuda_device, 64, 2)
    stage.middle = _Middle()
    x = torch.randn(4096, 64, device=cuda_device).bfloat16()
    first, _ = _both(stage, x)
    with torch.no_grad():
        stage.encoder_blocks[0].mlp.mlp.fc1_weight.mul_(1.5)          # in place, as an optimizer step
    a, b = _both(stage, x)
    assert torch.equal(a, b) and not torch.equal(a, first)
    stage.decoder_blocks[1].bwa.proj = torch.nn.Linear(64, 64).to(cuda_device)
    c, d = _both(stage, x)
    assert torch.equal(c, d) and not torch.equal(c, a)
    twin = copy.deepcopy(stage)
    assert torch.equal(_both(twin, x)[0], c)
    seen = []
    handle = stage.encoder_blocks[1].register_forward_hook(lambda m, i, o: seen.append(o.shape))
    assert torch.equal(_both(stage, x)[0], c) and len(seen) == 2      # the hook fires either way
    handle.remove()
    y = stage(None, x.float().requires_grad_(True), None)             # autograd: block by block
    y.float().sum().backward()
    assert stage.encoder_blocks[0].norm.weight.grad is not None


@pytest.mark.parametrize("c,rows,hd", [(32, 512, 16), (32, 4096, 32), (64, 4608, 32), (256, 1024, 32), (512, 1024, 64)])
def test_block_as_one_autograd_node(cuda_device, c, rows, hd):
    """Output and every gradient of the native block against the layers taken one by one (c = 512: weights past the native
    weight gradient's limit)."""
    from flash3dtransformer_b200.layers import stage as st
    stage = _stage(cuda_device, c, 1, hd)
    block = stage.encoder_blocks[0]
    x = torch.randn(rows, c, device=cuda_device).bfloat16()
    g = torch.randn(rows, c, device=cuda_device).bfloat16()
    got = []
    for native in (True, False):
        st.BlockStack.ENABLED = native
        try:
            block.zero_grad()
            xx = x.clone().requires_grad_(True)
            out = block(None, xx, None)
            assert (type(out.grad_fn).__name__ == "XfmrBlockFunctionBackward") == native
            out.backward(g)
        finally:
            st.BlockStack.ENABLED = True
        got.append([out.detach(), xx.grad] + [p.grad for p in block.parameters()])
    assert torch.equal(got[0][0], got[1][0])
    for a, b in zip(*got):
        assert a.dtype == b.dtype and (a.float() - b.float()).norm() <= 1e-2 * b.float().norm() + 1e-6
