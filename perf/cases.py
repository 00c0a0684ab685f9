"""The work that users have this framework do, as cases that can be timed.

The solver is used through one handle per problem (``capi.Solver``): a program
sets a problem, then evaluates the objective at trial weights, runs a solve
from the weights that it has (zero, the previous outer iteration's, a coarser
level's), and reads centroids at the end.  Warm starts add the damped Newton
solve on problems that change from call to call, batches of small instances,
and the network that predicts start weights, which is trained here too.

Sizes are those of this repository's problem generator (``problems.make``:
1,024 to 262,144 sites, images of 128^2 to 2048^2) and odd ones between them.
The weights are the ones that an optimal transport between the products of the
two sides' marginals gives, plus noise at the scale of the pitch: cells as far
from their sites, and as uneven in area, as they are well into a solve.  With
``warm`` the image is nearly such a product, so that they are also close to the
solution, as a coarser level's are; a cold solve starts from zero.

Solves are bounded by their iteration count, as ``total_iter`` bounds them in a
settings file, so that a pass is a fixed amount of work.
"""
import math

import numpy as np
import torch

from caustic_b200 import capi, warmstart

UNIT = (0.0, 1.0, 0.0, 1.0)
WIDE = (0.0, 160.0, -60.0, 100.0)  # the projection domain of the committed run's settings


def listed():
    return [
        # a small problem from numpy arrays: launches, copies and host work
        dict(name="eval 1k host", kind="eval", gx=32, gy=32, nx=128, ny=128, k=8, beam=False,
             wide=False, warm=False, device=False),
        # nothing square, nothing a power of two, a domain away from the origin
        dict(name="eval 12k ragged", kind="eval", gx=97, gy=131, nx=333, ny=245, k=7, beam=True,
             wide=True, warm=False, device=True),
        # the headline problem's evaluation, tensors on the GPU
        dict(name="eval 65k", kind="eval", gx=256, gy=256, nx=1024, ny=1024, k=16, beam=True,
             wide=False, warm=False, device=True),
        # the largest problem: 262,144 sites on a 2048^2 image
        dict(name="eval 262k", kind="eval", gx=512, gy=512, nx=2048, ny=2048, k=24, beam=True,
             wide=False, warm=True, device=True),
        # the first iterations of a cold solve (weights 0) of a small problem, numpy in and out
        dict(name="lbfgs 4k host", kind="lbfgs", gx=64, gy=64, nx=256, ny=256, k=8, beam=False, wide=False, warm=False,
             device=False, iters=25),
        # iterations late in a solve of the headline problem, device resident
        dict(name="lbfgs 65k", kind="lbfgs", gx=256, gy=256, nx=1024, ny=1024, k=16, beam=True, wide=False, warm=True,
             device=True, iters=15),
        # one level of the warm pipeline: a new problem in a kept handle, then the damped Newton solve
        dict(name="newton 16k", kind="newton", gx=128, gy=128, nx=256, ny=256, k=9, beam=False, wide=False, warm=True,
             tol=1e-4),
        # many small instances in one launch
        dict(name="batch 12", kind="batch", count=12, gx=32, gy=90, nx=512, ny=512, k=8, beam=False,
             wide=False, warm=False, iters=12),
        # the centroids that the lens fit reads (out.txt), once per outer iteration
        dict(name="centroids 65k", kind="centroids", gx=256, gy=256, nx=1024, ny=1024, k=16, beam=True,
             wide=False, warm=True),
        # the later outer iterations: masses re-weighted by the light path, Anderson acceleration
        dict(name="aarl 16k", kind="aarl", gx=128, gy=128, nx=256, ny=256, k=8, beam=False,
             wide=False, warm=True, iters=4),
        # the network's prediction for one problem on its 64^2 lattice, the warm pipeline's start
        dict(name="net forward 1x64", kind="forward", batch=1, gx=64, gy=64, levels=4, base=32),
        # one accumulation step of the training loop at its default batch on 128^2 lattices
        dict(name="net gradients 16x128", kind="gradients", batch=16, gx=128, gy=128, levels=4, base=32),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["eval", "eval", "eval", "lbfgs", "lbfgs", "newton", "batch", "centroids", "aarl", "forward",
                       "gradients"])
    if kind in ("forward", "gradients"):
        levels = rng.choice([3, 4])
        step = 2 ** (levels - 1)
        return dict(kind=kind, batch=log_int(1, 16), gx=step * log_int(24 // step, 128 // step),
                    gy=step * log_int(24 // step, 128 // step), levels=levels, base=32)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 16), gx=32, gy=log_int(36, 90), nx=log_int(200, 512),
                    ny=log_int(200, 512), k=rng.randint(4, 16), beam=False,
                               wide=False, warm=False, iters=rng.randint(4, 12))
    top = dict(eval=512, lbfgs=256, newton=160, centroids=256, aarl=128)[kind]
    gx = log_int(30, top)
    gy = min(top, max(24, int(gx * math.exp(rng.uniform(-0.5, 0.5)))))
    per = math.exp(rng.uniform(math.log(1.5), math.log(6.0)))  # pixels across a pitch
    cap = 2048 if kind == "eval" else 1024
    c = dict(kind=kind, gx=gx, gy=gy, nx=min(cap, int(gx * per)), ny=min(cap, int(gy * per)), k=rng.randint(2, 24),
             beam=rng.random() < 0.5, wide=rng.random() < 0.3, warm=kind in ("newton", "aarl") or rng.random() < 0.5)
    if kind in ("eval", "lbfgs"):
        c["device"] = rng.random() < 0.6
    if kind == "lbfgs":
        c["iters"] = rng.randint(5, 15)
    if kind == "newton":
        c["tol"] = rng.choice([1e-3, 1e-4])
    if kind == "aarl":
        c["iters"] = rng.randint(1, 4)
    return c


# -- problems -----------------------------------------------------------------


class Problem:
    """Sites on a jittered lattice, masses, a Gaussian-mixture image, and the
    weights of the separable transport (tensors on the GPU, float64)."""

    def __init__(self, rng, gx, gy, nx, ny, k, beam, wide, warm=True):
        dev = torch.device("cuda")
        self.grid, self.size = (gx, gy), (nx, ny)
        self.domain = np.array(WIDE if wide else UNIT)
        ex, ey = self.domain[1] - self.domain[0], self.domain[3] - self.domain[2]
        jit = torch.from_numpy(rng.uniform(-0.25, 0.25, size=(gy, gx, 2))).to(dev)
        a = torch.arange(gx, dtype=torch.float64, device=dev)
        b = torch.arange(gy, dtype=torch.float64, device=dev)
        ux = (a[None, :] + 0.5 + jit[..., 0]) / gx
        uy = (b[:, None] + 0.5 + jit[..., 1]) / gy
        img = self._image(rng, k, nx, ny, dev)
        sigma = 0.35
        mx = torch.exp(-((a + 0.5) / gx - 0.5) ** 2 / (2 * sigma**2)) if beam else torch.ones_like(a)
        my = torch.exp(-((b + 0.5) / gy - 0.5) ** 2 / (2 * sigma**2)) if beam else torch.ones_like(b)
        nu = my[:, None] * mx[None, :]
        if warm:
            # nine parts in ten the product of its marginals: the weights below are then near the solution
            img = img / img.sum()
            img = 0.9 * img.sum(1)[:, None] * img.sum(0)[None, :] + 0.1 * img
        w = self._axis_weights(mx, img.sum(0), ux) * ex**2 + self._axis_weights(my, img.sum(1), uy) * ey**2
        pitch2 = (ex / gx) * (ey / gy)
        noise = torch.from_numpy(rng.normal(0.0, 0.01, size=(2, gy, gx))).to(dev) * pitch2
        self.xy = torch.stack([self.domain[0] + ex * ux, self.domain[2] + ey * uy], -1).reshape(-1, 2).contiguous()
        self.nu = (nu / nu.sum() * (ex * ey)).reshape(-1).contiguous()
        self.density = (img / img.sum()).reshape(-1).contiguous()
        self.w0 = (w + noise[0]).reshape(-1).contiguous()
        self.w1 = (w + noise[0] + noise[1]).reshape(-1).contiguous()
        self.zero = torch.zeros_like(self.w0)
        self.n = gx * gy

    @staticmethod
    def _image(rng, k, nx, ny, dev):
        ctr = rng.uniform(0.1, 0.9, size=(k, 2))
        sig = rng.uniform(0.02, 0.15, size=(k, 2))
        th = rng.uniform(0.0, np.pi, size=k)
        amp = rng.uniform(0.2, 1.0, size=k)
        px = ((torch.arange(nx, dtype=torch.float64, device=dev) + 0.5) / nx)[None, :]
        py = ((torch.arange(ny, dtype=torch.float64, device=dev) + 0.5) / ny)[:, None]
        img = torch.full((ny, nx), 1e-3, dtype=torch.float64, device=dev)
        for c in range(k):
            dx, dy = px - ctr[c, 0], py - ctr[c, 1]
            ct, st = math.cos(th[c]), math.sin(th[c])
            img += amp[c] * torch.exp(-0.5 * (((ct * dx + st * dy) / sig[c, 0]) ** 2 +
                                              ((ct * dy - st * dx) / sig[c, 1]) ** 2))
        return img

    @staticmethod
    def _axis_weights(mass, target, u):
        """Weights of the transport of `mass` (on equal strips of [0, 1]) to
        `target`, at positions u: w' = 2 (s - T(s))."""
        m, t = mass.cpu().numpy(), target.cpu().numpy()
        s = np.linspace(0.0, 1.0, 16 * len(m) + 1)
        cm = np.concatenate([[0.0], np.cumsum(m) / m.sum()])
        ct = np.concatenate([[0.0], np.cumsum(t) / t.sum()])
        T = np.interp(np.interp(s, np.linspace(0, 1, len(m) + 1), cm), ct, np.linspace(0, 1, len(t) + 1))
        g = 2.0 * (s - T)
        h = s[1] - s[0]
        w = np.concatenate([[0.0], np.cumsum(0.5 * h * (g[1:] + g[:-1]))])
        # cubic in every strip: value and slope at both ends
        x = u.cpu().numpy().ravel() / h
        i = np.minimum(x.astype(np.int64), len(s) - 2)
        f = x - i
        v = (w[i] * (1 + 2 * f) * (1 - f) ** 2 + w[i + 1] * f * f * (3 - 2 * f) +
             h * (g[i] * f * (1 - f) ** 2 - g[i + 1] * f * f * (1 - f)))
        return torch.from_numpy(v.reshape(tuple(u.shape))).to(u.device)

    def host(self):
        for name in ("xy", "nu", "density", "w0", "w1", "zero"):
            setattr(self, name, getattr(self, name).cpu().numpy())
        return self


def _rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _problem(case, rng):
    return Problem(rng, *(case[k] for k in ("gx", "gy", "nx", "ny", "k", "beam", "wide", "warm")))


def _set(solver, p):
    solver.set_problem(p.xy, p.nu, p.density, p.size, p.domain)
    return solver


def _batch(case, rng):
    """Instances of config 3's kind: lattices of sizes spread from gx to gy."""
    out = []
    for i in range(case["count"]):
        # the sizes a case has are its own, in an order that does not follow them
        q = (i * 0.6180339887) % 1.0
        g = int(round(case["gx"] * (case["gy"] / case["gx"]) ** q))
        out.append(_problem(dict(case, gx=g, gy=g), rng))
    return out


# -- the network ----------------------------------------------------------------


def _net_weights(case, rng):
    """He-initialised convolutions of WarmStartNet's layer list, small biases."""
    ch = [case["base"] * 2**l for l in range(case["levels"])]
    shapes, cin = [], warmstart.IN_CH
    for c in ch:
        shapes += [(c, cin, 3), (c, c, 3)]
        cin = c
    for l in range(case["levels"] - 2, -1, -1):
        shapes += [(ch[l], ch[l + 1] + ch[l], 3), (ch[l], ch[l], 3)]
    sd = {"out_scale": 1.0}
    for k, (co, ci, s) in enumerate(shapes):
        sd["w%d" % k] = (rng.standard_normal((co, s * s * ci)) * math.sqrt(2.0 / (s * s * ci))).astype(np.float32)
        sd["b%d" % k] = (0.05 * rng.standard_normal(co)).astype(np.float32)
    head = np.zeros((8, ch[0]), np.float32)
    head[0] = rng.standard_normal(ch[0]) / math.sqrt(ch[0])
    sd["w%d" % len(shapes)] = head
    return sd


def _net_inputs(case, rng):
    """Inputs and targets as make_input / make_target lay them out: the
    log-density on the site grid, the sites' jitter, the log masses."""
    dev = torch.device("cuda")
    B, gx, gy = case["batch"], case["gx"], case["gy"]
    x = torch.zeros(B, gy, gx, warmstart.IN_CH, dtype=torch.float64, device=dev)
    y = torch.empty(B, gy * gx, dtype=torch.float64, device=dev)
    for b in range(B):
        p = Problem(rng, gx, gy, gx, gy, int(rng.integers(2, 17)), b % 4 != 3, False)
        lg = torch.log(p.density.view(gy, gx) * (gx * gy))
        x[b, ..., 0] = lg - lg.mean()
        xy = p.xy.view(gy, gx, 2)
        x[b, ..., 1] = (xy[..., 0] * gx - torch.arange(gx, device=dev) - 0.5) * 4
        x[b, ..., 2] = (xy[..., 1] * gy - torch.arange(gy, device=dev)[:, None] - 0.5) * 4
        x[b, ..., 3] = torch.log(p.nu.view(gy, gx) * p.n)
        y[b] = p.w0 * p.n
    y -= y.mean(1, keepdim=True)
    return x.to(torch.bfloat16), (y / y.std()).float()


# -- the cases ------------------------------------------------------------------


class State:
    pass


def prepare(case, seed):
    rng = _rng(seed)
    s = State()
    s.case = case
    kind = case["kind"]
    if kind in ("forward", "gradients"):
        s.net = warmstart.WarmStartNet(levels=case["levels"], base=case["base"])
        s.net.load_state_dict(_net_weights(case, rng))
        s.x, s.y = _net_inputs(case, rng)
        return s
    if kind == "batch":
        s.p = [p.host() for p in _batch(case, rng)]
        s.solvers = [_set(capi.Solver(), p) for p in s.p]
        return s
    s.p = _problem(case, rng)
    if kind == "aarl" or not case.get("device", True):
        s.p.host()
    s.solver = _set(capi.Solver(), s.p)
    if kind == "aarl":
        n = s.p.n
        inside = np.column_stack([rng.normal(0, 0.05, n), rng.normal(0, 0.05, n), np.ones(n)])
        s.inside = inside / np.linalg.norm(inside, axis=1, keepdims=True)
        s.light = np.tile([0.0, 0.0, 1.0], (n, 1))
        s.height = rng.uniform(5, 10, n)
        s.points = s.p.xy * 1.0
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "eval":
        # two trial points of a line search
        return [s.solver.eval(s.p.w0), s.solver.eval(s.p.w1)]
    if kind == "lbfgs":
        w, st = s.solver.solve(s.p.w0 if case["warm"] else s.p.zero, history=10, max_iter=case["iters"], tol=1e-9)
        return [w, st.f]
    if kind == "newton":
        _set(s.solver, s.p)
        w, st = s.solver.solve_newton(s.p.w0, tol=case["tol"])
        return [w - w.mean(), st.converged]  # weights are defined up to a constant
    if kind == "batch":
        ws, _ = capi.solve_batch(s.solvers, [p.zero for p in s.p], history=10, max_iter=case["iters"], tol=1e-9)
        return ws
    if kind == "centroids":
        return list(s.solver.centroids(s.p.w0))
    if kind == "aarl":
        # the problem's masses come back re-weighted: a caller sets the source masses again
        _set(s.solver, s.p)
        w, st = s.solver.solve_aarl(s.p.w0, s.points, s.light, s.inside, s.height, z_of_len=0.0, z_of_receiver=30.0,
                                    refraction_index=1.49, sample_domain=s.p.domain, aa_fixed_para=-0.1,
                                    max_iter=case["iters"], tol=1e-12)
        return [w, st.f]
    if kind == "forward":
        return s.net.forward(s.x)
    if kind == "gradients":
        s.net.zero_grad()
        pred = s.net.forward(s.x, keep=True)
        loss, g = s.net.loss_grad(pred, s.y, grid=(case["gy"], case["gx"]))
        s.net.backward(g)
        return [pred, loss, [c.gw for c in s.net.layers()], [c.gb for c in s.net.layers() if c.gb is not None]]
    raise ValueError(kind)


def work(case):
    kind = case["kind"]
    if kind in ("forward", "gradients"):
        px = case["batch"] * case["gx"] * case["gy"]
        ch = [case["base"] * 2**l for l in range(case["levels"])]
        flops, nbytes, cin = 0.0, 0.0, 4
        convs = []
        for l, c in enumerate(ch):
            convs += [(l, cin, c), (l, c, c)]
            cin = c
        for l in range(case["levels"] - 2, -1, -1):
            convs += [(l, ch[l + 1] + ch[l], ch[l]), (l, ch[l], ch[l])]
        for l, ci, co in convs:
            flops += 2.0 * 9 * ci * co * px / 4**l
            nbytes += 2.0 * 9 * ci * co
        io = px * (16 + 4)
        if kind == "forward":
            return {"bytes": nbytes + io, "flops": flops}
        # activations are kept for the backward pass; weight and input gradients are two more products
        acts = sum(2.0 * co * px / 4**l for l, _, co in convs)
        return {"bytes": 4 * nbytes + 2 * acts + io, "flops": 3 * flops}
    if kind == "batch":
        n = case["count"] * case["gx"] * case["gy"]  # the middle of the instances' sizes
        pixels = case["count"] * case["nx"] * case["ny"]
    else:
        n, pixels = case["gx"] * case["gy"], case["nx"] * case["ny"]
    per = pixels / n
    # one evaluation: sites, weights and masses in, masses and objective out, the density once; per cell six
    # vertices (20), six sides tested against the ring (36 x 4), and an integral term for each piece of the
    # boundary and each pixel column inside (30 each)
    ev = {"bytes": 8.0 * pixels + 56.0 * n, "flops": n * (270.0 + 30.0 * (6 + 4 * math.sqrt(per) + per))}
    times = {"eval": 2, "lbfgs": case.get("iters", 0) + 1, "newton": 4,
             "batch": case.get("iters", 0) + 1, "centroids": 1, "aarl": 2 * case.get("iters", 0) + 3}[kind]
    out = {"bytes": times * ev["bytes"], "flops": times * ev["flops"]}
    if kind in ("lbfgs", "batch", "aarl"):
        out["bytes"] += 8.0 * n * 46 * case["iters"]  # the history of ten pairs, read twice
        out["flops"] += 4.0 * n * 40 * case["iters"]
    return out


# -- the same results in plain torch ----------------------------------------------


def _clip(X, Y, n, a, b, c):
    """Convex polygons (rows of X, Y; n vertices each) cut by a x + b y <= c."""
    m, V = X.shape
    k = torch.arange(V, device=X.device)[None, :]
    valid = k < n[:, None]
    nxt = torch.where(k + 1 < n[:, None], k + 1, torch.zeros_like(k)).expand(m, V)
    d = a[:, None] * X + b[:, None] * Y - c[:, None]
    dn = d.gather(1, nxt)
    ins = valid & (d <= 0)
    cross = valid & ((d <= 0) != (dn <= 0))
    t = torch.where(cross, d / torch.where(cross, d - dn, torch.ones_like(d)), torch.zeros_like(d))
    cnt = ins.long() + cross.long()
    pos = cnt.cumsum(1) - cnt
    trash = torch.full_like(pos, V)
    oX = torch.zeros(m, V + 1, dtype=X.dtype, device=X.device)
    oY = torch.zeros_like(oX)
    p1 = torch.where(ins, pos, trash).clamp(max=V)
    p2 = torch.where(cross, pos + ins.long(), trash).clamp(max=V)
    oX.scatter_(1, p1, X)
    oY.scatter_(1, p1, Y)
    oX.scatter_(1, p2, X + t * (X.gather(1, nxt) - X))
    oY.scatter_(1, p2, Y + t * (Y.gather(1, nxt) - Y))
    return oX[:, :V], oY[:, :V], cnt.sum(1).clamp(max=V)


def _rings(p, w, V=24, reach=8):
    """Power cells inside the domain, relative to their sites; None when the
    sites within `reach` lattice steps do not bound them all."""
    gx, gy = p.grid
    x, y = p.xy[:, 0], p.xy[:, 1]
    d = p.domain
    X = torch.zeros(p.n, V, dtype=torch.float64, device=x.device)
    Y = torch.zeros_like(X)
    X[:, 0], X[:, 1], X[:, 2], X[:, 3] = d[0] - x, d[1] - x, d[1] - x, d[0] - x
    Y[:, 0], Y[:, 1], Y[:, 2], Y[:, 3] = d[2] - y, d[2] - y, d[3] - y, d[3] - y
    n = torch.full((p.n,), 4, dtype=torch.long, device=x.device)
    i = torch.arange(p.n, device=x.device)
    ia, ib = i % gx, i // gx
    steps = sorted(((u * u + v * v, u, v) for u in range(-reach, reach + 1) for v in range(-reach, reach + 1)
                    if u or v))
    for _, u, v in steps:
        ok = (ia + u >= 0) & (ia + u < gx) & (ib + v >= 0) & (ib + v < gy)
        j = torch.where(ok, i + u + v * gx, i)
        a, b = x[j] - x, y[j] - y
        c = 0.5 * (a * a + b * b - (w[j] - w))
        X, Y, n = _clip(X, Y, n, a, b, c)
    area = _moments(X, Y, n)[0]
    whole = (d[1] - d[0]) * (d[3] - d[2])
    if int(n.max()) >= V or abs(float(area.sum()) / whole - 1) > 1e-11:
        return None
    return X, Y, n


def _moments(X, Y, n):
    """Integrals of 1, x, y, x^2 + y^2 over the polygons."""
    m, V = X.shape
    k = torch.arange(V, device=X.device)[None, :]
    valid = k < n[:, None]
    nxt = torch.where(k + 1 < n[:, None], k + 1, torch.zeros_like(k)).expand(m, V)
    X1, Y1 = X.gather(1, nxt), Y.gather(1, nxt)
    cr = torch.where(valid, X * Y1 - X1 * Y, torch.zeros_like(X))
    return (cr.sum(1) / 2, (cr * (X + X1)).sum(1) / 6, (cr * (Y + Y1)).sum(1) / 6,
            (cr * (X * X + X * X1 + X1 * X1 + Y * Y + Y * Y1 + Y1 * Y1)).sum(1) / 12)


def _integrate(p, w, smallest=0.0):
    """Per cell: integrals of the scaled density times 1, x, y, |x - s|^2
    (coordinates relative to the site) over pieces above `smallest` in area,
    and the cell's area; None when the cells could not be built."""
    rings = _rings(p, w)
    if rings is None:
        return None
    X, Y, n = rings
    nx, ny = p.size
    d = p.domain
    sx, sy = (d[1] - d[0]) / nx, (d[3] - d[2]) / ny
    rho = p.density * (p.nu.sum() / p.density.sum()) / (sx * sy)
    k = torch.arange(X.shape[1], device=X.device)[None, :]
    some = k < n[:, None]
    inf = float("inf")

    def box(Z, s, lo, step, cells):
        a = torch.where(some, Z, torch.full_like(Z, inf)).min(1)[0] + s
        b = torch.where(some, Z, torch.full_like(Z, -inf)).max(1)[0] + s
        c0 = torch.floor((a - lo) / step).clamp(0, cells - 1).nan_to_num(0)
        c1 = torch.floor((b - lo) / step).clamp(0, cells - 1).nan_to_num(-1)
        return c0.long(), torch.where(n >= 3, c1.long() - c0.long() + 1, torch.zeros_like(n))

    def wide(Z):  # room for the four cuts
        return torch.nn.functional.pad(Z, (0, 4))

    x0, wx = box(X, p.xy[:, 0], d[0], sx, nx)
    y0, wy = box(Y, p.xy[:, 1], d[2], sy, ny)
    cnt = wx * wy
    acc = torch.zeros(4, p.n, dtype=torch.float64, device=X.device)
    ends = cnt.cumsum(0)
    start = 0
    while start < p.n:
        done = int(ends[start - 1]) if start else 0
        stop = max(start + 1, int(torch.searchsorted(ends, done + 800_000, right=True)))
        i = torch.repeat_interleave(torch.arange(start, stop, device=X.device), cnt[start:stop])
        q = torch.arange(len(i), device=X.device) + done - (ends - cnt)[i]
        ix, iy = x0[i] + q % wx[i].clamp(min=1), y0[i] + q // wx[i].clamp(min=1)
        cx = d[0] + (ix.double() + 0.5) * sx - p.xy[i, 0]
        cy = d[2] + (iy.double() + 0.5) * sy - p.xy[i, 1]
        PX, PY, m = wide(X)[i] - cx[:, None], wide(Y)[i] - cy[:, None], n[i]
        one = torch.ones_like(cx)
        for a, b, c in ((1, 0, sx / 2), (-1, 0, sx / 2), (0, 1, sy / 2), (0, -1, sy / 2)):
            PX, PY, m = _clip(PX, PY, m, a * one, b * one, c * one)
        A, Mx, My, M2 = _moments(PX, PY, m)
        r = torch.where(A > smallest, rho[ix + iy * nx], torch.zeros_like(A))
        acc[0].index_add_(0, i, r * A)
        acc[1].index_add_(0, i, r * (Mx + cx * A))
        acc[2].index_add_(0, i, r * (My + cy * A))
        acc[3].index_add_(0, i, r * (M2 + 2 * (cx * Mx + cy * My) + (cx * cx + cy * cy) * A))
        start = stop
    return acc, _moments(X, Y, n)[0]


def _exact_eval(p, w):
    got = _integrate(p, w)
    if got is None:
        return None
    (mu, _, _, m2), _ = got
    fc = w * (mu - p.nu) - m2
    return [float(fc.sum()), mu, mu - p.nu, fc]


def _exact_net(case, rng, gradients):
    F = torch.nn.functional
    sd = _net_weights(case, rng)
    x, y = _net_inputs(case, rng)
    dev = x.device
    L = case["levels"]
    nconv = 2 * L + 2 * (L - 1)
    W = [torch.from_numpy(sd["w%d" % k]).to(dev).double().requires_grad_() for k in range(nconv + 1)]
    b = [torch.from_numpy(sd["b%d" % k]).to(dev).double().requires_grad_() for k in range(nconv)]

    def conv(k, h):
        w = W[k].view(W[k].shape[0], 3, 3, -1).permute(0, 3, 1, 2)
        return F.relu(F.conv2d(h, w, b[k], padding=1))

    with torch.set_grad_enabled(gradients):
        h = x.double().permute(0, 3, 1, 2)
        k, skips = 0, []
        for l in range(L):
            h = conv(k + 1, conv(k, h))
            k += 2
            skips.append(h)
            if l < L - 1:
                h = F.avg_pool2d(h, 2)
        for l in range(L - 2, -1, -1):
            h = torch.cat([F.interpolate(h, scale_factor=2, mode="nearest"), skips[l]], 1)
            h = conv(k + 1, conv(k, h))
            k += 2
        pred = torch.einsum("bchw,c->bhw", h, W[nconv][0]).reshape(x.shape[0], -1)
        if not gradients:
            return pred
        e = pred - y.double()
        e = e - e.mean(1, keepdim=True)
        loss = (e * e).sum() / e.numel()
        loss.backward()
    return [pred.detach(), float(loss.detach()), [v.grad for v in W], [v.grad for v in b]]


def exact(case, seed):
    kind = case["kind"]
    rng = _rng(seed)
    if kind in ("forward", "gradients"):
        return _exact_net(case, rng, kind == "gradients")
    if kind == "eval":
        p = _problem(case, rng)
        both = [_exact_eval(p, p.w0), _exact_eval(p, p.w1)]
        return None if both[0] is None or both[1] is None else both
    if kind == "centroids":
        p = _problem(case, rng)
        got = _integrate(p, p.w0, smallest=1e-10)  # the reference leaves out smaller pieces
        if got is None:
            return None
        (m, mx, my, _), _ = got
        if not bool((m > 0).all()):
            return None
        return [torch.stack([p.xy[:, 0] + mx / m, p.xy[:, 1] + my / m], -1), None]
    return None  # a solve of many steps: its value is the sequence of its own evaluations
