"""The network's fused layers (one GEMM with bias and ReLU in its epilogue, no
concatenated or upsampled tensor, weight gradients on side streams) against
the same network run launch by launch, as a trace makes it run."""
import numpy as np
import pytest

from caustic_b200 import warmstart

pytestmark = pytest.mark.gpu


def build(torch, levels, base, seed):
    net = warmstart.WarmStartNet(levels=levels, base=base, seed=seed)
    g = torch.Generator(device="cpu").manual_seed(seed)
    for c in net.layers():
        if c.b is not None:
            c.b.copy_(0.1 * torch.randn(c.cout, generator=g))
    return net


# one tile and several, widths that are no power of two, channel counts on both
# sides of the tile widths, an image of one pixel at the deepest level
@pytest.mark.parametrize("levels,base,B,H,W", [
    (3, 8, 2, 16, 16), (3, 32, 2, 24, 40), (4, 32, 8, 8, 8), (2, 64, 1, 34, 16), (1, 16, 3, 8, 15), (3, 40, 8, 12, 20),
])
def test_fused_layers_have_the_bits_of_the_single_launches(gpu, levels, base, B, H, W):
    import torch

    rng = np.random.default_rng(H * W)
    x = torch.from_numpy(rng.normal(size=(B, H, W, warmstart.IN_CH)).astype(np.float32)).cuda().to(torch.bfloat16)
    t = torch.from_numpy(rng.normal(size=(B, H * W)).astype(np.float32)).cuda()
    out = []
    for traced in (True, False):
        net = build(torch, levels, base, 7)
        net.trace = [] if traced else None
        net.zero_grad()
        pred = net.forward(x, keep=True)
        loss, g = net.loss_grad(pred, t, grid=(H, W), lam=0.5)
        dx = net.backward(g)
        torch.cuda.synchronize()
        out.append((pred, loss, dx, [c.gw for c in net.layers()], [c.gb for c in net.layers() if c.gb is not None]))
        # a prediction alone keeps nothing and gives the same
        assert torch.equal(net.forward(x), pred)
    a, b = out
    assert torch.equal(a[0], b[0]) and a[1] == b[1] and torch.equal(a[2], b[2])
    for u, v in zip(a[3], b[3]):
        assert torch.equal(u, v)
    # fp32 sums of at most 2,720 terms in another order
    for u, v in zip(a[4], b[4]):
        assert float((u - v).norm()) <= 1e-5 * float(u.norm())
