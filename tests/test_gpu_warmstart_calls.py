"""Ways of calling the network that its fused layers have to bear: streams of
the caller's choice, a trace set late, layers that are not plain."""
import numpy as np
import pytest

from caustic_b200 import warmstart
from test_gpu_warmstart_fused import build

pytestmark = pytest.mark.gpu

SHAPE = (4, 32, 32)


def inputs(torch, seed=0):
    B, H, W = SHAPE
    rng = np.random.default_rng(seed)
    x = torch.from_numpy(rng.normal(size=(B, H, W, warmstart.IN_CH)).astype(np.float32)).cuda().to(torch.bfloat16)
    g = torch.from_numpy(rng.normal(size=(B, H * W)).astype(np.float32)).cuda()
    return x, g


def gradients(net):
    return [t for c in net.layers() for t in (c.gw, c.gb) if t is not None]


def test_backward_on_another_stream(gpu):
    """The tape is forward()'s memory: backward() on another stream waits for
    it, and gives it back only when it has been read."""
    import torch

    x, g = inputs(torch)
    net = build(torch, 3, 32, 5)
    net.zero_grad()
    net.forward(x, keep=True)
    want_dx = net.backward(g)
    torch.cuda.synchronize()
    want = [t.clone() for t in gradients(net)]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    net.zero_grad()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(100_000_000)  # forward() is far from done when backward() is called
        net.forward(x, keep=True)
        sizes = [t.numel() * t.element_size() for e in net._tape[0] for t in e[1:3] if t is not None]
    with torch.cuda.stream(b):
        torch.cuda._sleep(100_000_000)  # and backward() when forward()'s stream allocates again
        dx = net.backward(g)
    with torch.cuda.stream(a):
        over = [torch.full((n,), 0x7f, dtype=torch.uint8, device="cuda") for n in sizes]
    torch.cuda.synchronize()
    assert len(over) == len(sizes) and torch.equal(dx, want_dx)
    for u, v in zip(gradients(net), want):
        assert torch.equal(u, v)


def test_a_trace_set_after_the_forward_pass_is_recorded(gpu):
    import torch

    x, g = inputs(torch, 1)
    got = []
    for late in (False, True):
        net = build(torch, 3, 32, 5)
        net.zero_grad()
        net.trace = None if late else []
        net.forward(x, keep=True)
        net.trace = []
        net.backward(g)
        got.append(([[c is e[0] for c in net.layers()].index(True) for e in net.trace], [e[1:] for e in net.trace]))
    assert got[0][0] == got[1][0] and len(got[0][0]) == 11
    for u, v in zip(got[0][1], got[1][1]):
        for p, q in zip(u, v):
            assert torch.equal(p, q)


@pytest.mark.parametrize("what", ["no relu", "bias off a 16-byte boundary"])
def test_layers_that_the_fused_launch_does_not_take(gpu, what):
    """They run launch by launch, as a trace makes them."""
    import torch

    x, g = inputs(torch, 2)
    out = []
    for traced in (True, False):
        net = build(torch, 3, 32, 5)
        if what == "no relu":
            net.enc[1][0].relu = net.dec[0][1].relu = False
        else:
            c = net.dec[0][0]
            room = torch.zeros(c.cout + 1, device="cuda")
            room[1:].copy_(c.b)
            c.b = room[1:]
        net.trace = [] if traced else None
        net.zero_grad()
        pred = net.forward(x, keep=True)
        dx = net.backward(g)
        torch.cuda.synchronize()
        out.append([pred, dx] + gradients(net))
    for u, v in zip(*out):
        assert torch.equal(u, v)


def test_layer_refuses_addresses_that_its_vectors_do_not_fit(gpu):
    import torch

    L = warmstart.load()
    a, w = (torch.zeros(64, 72, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    y = torch.zeros(64, 64, dtype=torch.bfloat16, device="cuda")
    b = torch.zeros(64 + 4, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert L.ws_layer(64, 64, 72, a.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), s) == 0
    assert L.ws_layer(64, 64, 72, a.data_ptr(), w.data_ptr(), b.data_ptr() + 16, y.data_ptr(), s) == 0
    for args in ((a.data_ptr(), w.data_ptr(), b.data_ptr() + 4, y.data_ptr()),
                 (a.data_ptr() + 8, w.data_ptr(), b.data_ptr(), y.data_ptr()),
                 (a.data_ptr(), w.data_ptr() + 2, b.data_ptr(), y.data_ptr()),
                 (a.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr() + 2)):
        assert L.ws_layer(64, 64, 72, *args, s) == -1  # WS_EINVAL, before any launch
    torch.cuda.synchronize()


def test_gradients_pass_positive_values_below_the_smallest_bf16(gpu):
    """Pre-activations that are positive in fp32 and round to 0 in bf16 pass
    their gradient on, as the fp32 mask of the single launches has it."""
    import torch

    x, g = inputs(torch, 3)
    out = []
    for traced in (True, False):
        net = build(torch, 2, 16, 5)
        for c, r in ((net.enc[0][0], 0), (net.enc[1][1], 8), (net.dec[0][1], 1)):
            # rows of no weights: their pre-activations are the biases
            tiny = torch.tensor([1e-41, 2.0 ** -134, 5e-41, 0.0, -1e-41, 2.0 ** -133, 1.5e-38], device="cuda")
            c.w[r:r + 7] = 0.0
            c.w16[r:r + 7] = 0.0
            c.b[r:r + 7] = tiny
        net.trace = [] if traced else None
        net.zero_grad()
        pred = net.forward(x, keep=True)
        dx = net.backward(g)
        torch.cuda.synchronize()
        assert float(net.enc[0][0].gb[0].abs()) > 0.0 or not traced
        out.append([pred, dx] + gradients(net))
    for u, v in zip(*out):
        # the biases' gradients are fp32 sums in another order
        assert torch.equal(u, v) if u.dim() > 1 else float((u - v).norm()) <= 1e-5 * float(u.norm())
        assert torch.equal(u != 0, v != 0)
