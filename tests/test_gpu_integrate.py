"""The 8-lane integration (four cells a warp, problems above 4,096 sites)
against the oracle: pixel grids that cut the cells every way, cells aligned
with the pixels, rings around its capacity, boxes around its limits."""
import numpy as np
import pytest

from caustic_b200 import capi, problems
from oracle import oracle as O
from test_gpu_parity import check_eval, solver_for

pytestmark = pytest.mark.gpu

GX, GY = 73, 59  # 4,307 sites: not a multiple of four cells


def lattice(nx, ny, pd, jitter, seed):
    rng = np.random.default_rng(seed)
    u = (np.arange(GX) + 0.5 + rng.uniform(-jitter, jitter, (GY, GX))) / GX
    v = ((np.arange(GY) + 0.5)[:, None] + rng.uniform(-jitter, jitter, (GY, GX))) / GY
    xy = np.column_stack([pd[0] + (pd[1] - pd[0]) * u.ravel(), pd[2] + (pd[3] - pd[2]) * v.ravel()])
    nu = rng.uniform(0.5, 1.5, len(xy))
    pic = rng.uniform(0.0, 1.0, nx * ny) ** 2
    pic[rng.uniform(size=nx * ny) < 0.1] = 0.0
    p = problems.SDOTProblem("lattice", xy, nu / nu.sum(), pic / pic.sum(), (nx, ny), np.array(pd, float))
    return p, (pd[1] - pd[0]) * (pd[3] - pd[2]) / len(xy), rng


@pytest.mark.parametrize("nx,ny,pd,jitter", [
    (292, 236, [0.0, 1.0, 0.0, 1.0], 0.0),      # cell sides on pixel lines, four cells at a vertex
    (219, 118, [-3.3, 7.1, 0.7, 2.9], 0.0),     # sides half a pixel off the lines
    (301, 173, [0.0, 160.0, -60.0, 100.0], 0.3),
    (900, 41, [0.0, 1.0, 0.0, 1.0], 0.3),       # many lines one way, fewer than a row a cell the other
    (1, 1, [-1.0, 1.0, -1.0, 1.0], 0.3),
])
def test_small_cells_match_oracle(gpu, nx, ny, pd, jitter):
    p, cell, rng = lattice(nx, ny, pd, jitter, nx + ny)
    s = solver_for(p)
    for w in (np.zeros(p.n), rng.normal(0.0, 0.4 * cell, p.n)):
        check_eval(p, w, s)


def test_rings_and_boxes_around_the_limits(gpu):
    """A few strongly weighted sites among small ones: rings of more than 8
    and more than 16 edges, boxes below and above the limits of both paths."""
    p, cell, rng = lattice(584, 472, [0.0, 1.0, 0.0, 1.0], 0.3, 3)
    w = rng.normal(0.0, 0.1 * cell, p.n)
    big = rng.choice(p.n, 40, replace=False)
    w[big] += np.linspace(0.5, 40.0, 40) * cell
    s = solver_for(p)
    check_eval(p, w, s)
    off, _, _ = s.cells(w)
    sizes = np.diff(off)
    c = s.eval_counters()
    assert (sizes > 16).any() and ((sizes > 8) & (sizes <= 16)).any(), np.bincount(sizes)
    assert c["integrated_first"] > 0 and c["integrations_split"] > 0, c


@pytest.mark.parametrize("g,res", [(20, 1024), (40, 640), (72, 300)])
def test_pixel_parts_of_large_and_small_cells(gpu, g, res):
    """Weighted centroids and the render: cells that eight warps share (2,600
    pixels), that one warp takes (256) and that four share a warp for (17)."""
    p = problems.make(1, g=g, res=res)
    w = np.random.default_rng(g).normal(0.0, 0.1 / p.n, p.n)
    s = solver_for(p)
    xy, ex = s.centroids(w, weighted=True)
    c = O.cells(p.xy, w, O.proj_corner(p.xy, p.proj_domain))
    oxy, oex = O.centers(c, p.picture, p.size, p.proj_domain, weighting=True)
    assert np.array_equal(ex, oex)
    assert np.abs(xy[ex] - oxy[ex]).max() < 1e-10
    pxy, pex = s.centroids(w, weighted=False)
    oxy, oex = O.centers(c, p.picture, p.size, p.proj_domain, weighting=False)
    assert np.array_equal(pex, oex) and np.abs(pxy[pex] - oxy[pex]).max() < 1e-10
    # each cell's mass is spread over its pixels in proportion to area: the
    # whole is kept, and an all-equal density gives an even picture
    img = s.render(w)
    assert abs(img.sum() - p.nu.sum()) < 1e-10 * p.nu.sum()
    _, mu, _, _ = s.eval(w)
    flat = capi.Solver()
    flat.set_problem(p.xy, np.ones(p.n) / p.n, np.ones(res * res), p.size, p.proj_domain)
    area = flat.eval(w)[1] * 1.0
    flat.set_problem(p.xy, area, np.ones(res * res), p.size, p.proj_domain)
    img = flat.render(w)
    assert np.abs(img * res * res - 1.0).max() < 1e-9


@pytest.mark.parametrize("offset,width,k", [(3.0e3, 0.7, 4), (1.0e4, 1.9, 8), (1.0e5, 0.7, 4), (-1.0e5, 1.9, 5)])
def test_pixel_parts_of_aligned_cells_far_from_the_origin(gpu, offset, width, k):
    """Weighted centroids and the render where a cell's sides lie on pixel
    lines up to the coordinates' rounding, which is far above a pixel's own."""
    gx, gy = 32, 24
    nx, ny = k * gx, k * gy
    pd = np.array([offset, offset + width, 0.5 * offset, 0.5 * offset + width * gy / gx])
    X, Y = np.meshgrid(pd[0] + (np.arange(gx) + 0.5) * (pd[1] - pd[0]) / gx,
                       pd[2] + (np.arange(gy) + 0.5) * (pd[3] - pd[2]) / gy)
    rng = np.random.default_rng(k)
    nu = rng.uniform(0.5, 1.5, gx * gy)
    pic = rng.uniform(0.1, 1.0, nx * ny)
    s = capi.Solver()
    s.set_problem(np.column_stack([X.ravel(), Y.ravel()]), nu / nu.sum(), pic / pic.sum(), (nx, ny), pd)
    xy, ex = s.centroids(np.zeros(gx * gy), weighted=True)
    img = s.render(np.zeros(gx * gy))
    # each cell is k x k whole pixels
    rho = pic.reshape(gy, k, gx, k)
    at = (np.arange(k) + 0.5) / k
    mass = rho.sum((1, 3))
    wx = (np.arange(gx) + (rho * at).sum((1, 3)) / mass) * width / gx
    wy = (np.arange(gy)[:, None] + (rho * at[:, None, None]).sum((1, 3)) / mass) * width / gx
    # four sides a pixel, each at most four units in the last place of a
    # coordinate off its line
    ulp = np.spacing(np.abs(pd).max())
    rel = 16.0 * ulp / (width / nx)
    tol = rel * width / gx + 4.0 * ulp
    assert ex.all()
    assert np.abs(xy[:, 0] - pd[0] - wx.ravel()).max() <= tol
    assert np.abs(xy[:, 1] - pd[2] - wy.ravel()).max() <= tol
    want = np.repeat(np.repeat(nu.reshape(gy, gx) / nu.sum() / k ** 2, k, 0), k, 1)
    got = np.asarray(img).reshape(ny, nx)
    assert np.abs(got / want - 1.0).max() <= rel


@pytest.mark.parametrize("gx,gy,nx,ny", [(1, 1, 20, 30), (3, 2, 7, 9), (64, 64, 100, 90), (241, 17, 300, 31), (9, 7, 900, 700)])
def test_pixel_parts_at_the_sizes_where_the_form_changes(gpu, gx, gy, nx, ny):
    """Weighted centroids and the render up to 4,096 sites, a warp a cell, and
    just above, four cells a warp; cells that all go to eight warps."""
    rng = np.random.default_rng(gx + nx)
    xy = problems.jittered_grid(rng, gx, gy)
    n = gx * gy
    nu = rng.uniform(0.5, 1.5, n)
    p = problems.SDOTProblem("form", xy, nu / nu.sum(), rng.uniform(0.1, 1.0, nx * ny), (nx, ny))
    s = solver_for(p)
    for w in (np.zeros(n), rng.normal(0.0, 1.0 / n, n)):  # the second hides some cells
        c = O.cells(p.xy, w, O.proj_corner(p.xy, p.proj_domain))
        oxy, oex = O.centers(c, p.picture, p.size, p.proj_domain, weighting=True)
        for _ in range(2):  # without and with the cells of the call before
            got, ex = s.centroids(w, weighted=True)
            assert np.array_equal(ex, oex) and np.abs(got[ex] - oxy[ex]).max() < 1e-10
        oxy, oex = O.centers(c, p.picture, p.size, p.proj_domain, weighting=False)
        got, ex = s.centroids(w, weighted=False)
        assert np.array_equal(ex, oex) and np.abs(got[ex] - oxy[ex]).max() < 1e-10
        # the picture of the cells' masses: each cell's whole mass arrives
        img = s.render(w)
        assert abs(img.sum() - p.nu[ex].sum()) < 1e-10
