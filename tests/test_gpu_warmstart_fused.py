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
    (2, 520, 2, 4, 8), (2, 1032, 1, 4, 8),  # above 1,024 channels
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


def test_values_that_are_not_finite_pass_the_fused_layers_as_the_single_ones(gpu):
    """The ReLU of the single launches turns a NaN into 0."""
    import torch

    rng = np.random.default_rng(2)
    x = torch.from_numpy(rng.normal(size=(2, 16, 16, warmstart.IN_CH)).astype(np.float32)).cuda().to(torch.bfloat16)
    x[0, 3, 4, 1] = float("nan")
    x[1, 8, 9, 2] = float("inf")
    net = build(torch, 3, 32, 7)
    fused = net.forward(x)
    net.trace = []
    assert torch.equal(net.forward(x), fused)


def test_patches_above_the_pieces_of_one_launch(gpu):
    """Upsampled and skip channels of 2^30 pieces and more: whole images a
    launch, then bands of an image's rows.  Compared with the concatenation's
    patches at the seams."""
    import torch

    L = warmstart.load()
    # two images a launch at most, then one whose rows are split (9 * 2 pieces a pixel)
    for B, H, W in ((3, 5000, 5000), (1, 9000, 9000)):
        up = torch.randn(B, H // 2, W // 2, 8, device="cuda").to(torch.bfloat16)
        skip = torch.randn(B, H, W, 8, device="cuda").to(torch.bfloat16)
        cols = torch.empty(B * H * W, 9, 16, dtype=torch.bfloat16, device="cuda")
        assert L.ws_im2col_up(B, H, W, 8, up.data_ptr(), 8, skip.data_ptr(), cols.data_ptr(),
                              torch.cuda.current_stream().cuda_stream) == 0
        band = (1 << 30) // (W * 18)
        rows = {0, 1, H // 2, H - 1, min(H, band) - 1, min(H - 1, band), min(H - 1, band + 1)}
        pad = torch.nn.functional.pad
        for b in range(B):
            for y in rows:
                ys = [t for t in (y - 1, y, y + 1) if 0 <= t < H]
                part = torch.cat([up[b, [t // 2 for t in ys]].repeat_interleave(2, 1), skip[b, ys]], -1)
                part = pad(part, (0, 0, 1, 1, int(y == 0), int(y == H - 1)))
                want = torch.stack([part[q // 3, q % 3:q % 3 + W] for q in range(9)], 1)
                assert torch.equal(cols.view(B, H, W, 9, 16)[b, y], want), (b, y)
        del up, skip, cols
