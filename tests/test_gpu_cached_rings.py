"""Cells rebuilt from the last evaluation's ring and certified by a few lanes
(problems of at least 16,384 sites): the bits of an evaluation without a
cache, whichever cells the short path takes."""
import numpy as np
import pytest

from caustic_b200 import capi, problems
from test_gpu_parity import check_eval, solver_for

pytestmark = pytest.mark.gpu


# 8 lanes a cell and 4; sizes that leave a part of a block and of a tile of
# cells, and the last one below the short path
@pytest.mark.parametrize("gx,gy", [(128, 128), (141, 129), (223, 187), (131, 125)])
def test_cached_evaluation_has_the_bits_of_a_cold_one(gpu, gx, gy):
    rng = np.random.default_rng(gx)
    xy = problems.jittered_grid(rng, gx, gy)
    n = gx * gy
    nu = rng.uniform(0.5, 1.5, n)
    pic = problems.gaussian_mixture(rng, 6, 333, 290)
    p = problems.SDOTProblem("cached", xy, nu / nu.sum(), pic, (333, 290))
    s = solver_for(p)
    base = 0.3 / n * np.sin(7 * xy[:, 0]) * np.cos(5 * xy[:, 1]) * np.sqrt(n)
    w = base + rng.normal(0.0, 0.05 / n, n)
    # nothing moves, a few rings change, most change, cells hide and return
    for amp in (0.0, 0.01, 0.3, 3.0, 0.0):
        w = w + rng.normal(0.0, amp / n, n)
        f, mu, g, fc = s.eval(w)
        fresh = solver_for(p)
        f0, mu0, g0, fc0 = fresh.eval(w)
        assert np.array_equal(mu, mu0) and np.array_equal(fc, fc0) and f == f0, amp
        fresh.close()
    check_eval(p, base, s)


def test_jacobian_of_cached_rings(gpu):
    """The rows of cells finished by the short path: k_hessian reads their
    generators where k_rings_cached left them."""
    p = problems.make(4, g=129, res=200)
    rng = np.random.default_rng(3)
    w = rng.normal(0.0, 0.05 / p.n, p.n)
    warm = solver_for(p)
    warm.eval(w)
    warm.eval(w + rng.normal(0.0, 0.01 / p.n, p.n))
    a, b = warm.mass_jacobian(w), solver_for(p).mass_jacobian(w)
    assert np.array_equal(a.indptr, b.indptr) and np.array_equal(a.indices, b.indices)
    assert np.array_equal(a.data, b.data)


def test_domain_too_small_for_squares_in_single_precision(gpu):
    """A domain 2^-90 across: the short path's single-precision tests see only
    zeros there and leave every cell to the others."""
    p = problems.make(4, g=129, res=200)
    k = 2.0 ** -90
    small = problems.SDOTProblem("small", p.xy * k, p.nu * k * k, p.picture, p.size, np.asarray(p.proj_domain) * k)
    rng = np.random.default_rng(5)
    s = solver_for(small)
    w = np.zeros(p.n)
    for amp in (0.0, 0.05, 1.0):
        w = w + rng.normal(0.0, amp / p.n, p.n)
        _, mu, _, _ = s.eval(w * k * k)
        _, mu0, _, _ = solver_for(small).eval(w * k * k)
        assert np.array_equal(mu, mu0), amp


@pytest.mark.parametrize("n,width", [(16384, 0.01), (45000, 0.0005)])  # 8 lanes a cell, and 4
def test_clustered_sites_have_the_bits_of_a_cold_evaluation(gpu, n, width):
    """Half of the sites in a few buckets: leaves of more sites than the short
    path looks through go to the warp kernels."""
    rng = np.random.default_rng(n)
    xy = rng.uniform(0.0, 1.0, (n, 2))
    xy[: n // 2] = np.clip(0.5 + width * rng.normal(size=(n // 2, 2)), 0.0, 1.0)
    nu = rng.uniform(0.5, 1.5, n)
    pic = problems.gaussian_mixture(rng, 6, 128, 128)
    p = problems.SDOTProblem("clustered", xy, nu / nu.sum(), pic, (128, 128))
    s = solver_for(p)
    for amp in (0.0, 1e-3, 0.0):
        w = amp * width * width / n * rng.normal(size=n)
        f, mu, g, fc = s.eval(w)
        fresh = solver_for(p)
        f0, mu0, g0, fc0 = fresh.eval(w)
        assert np.array_equal(mu, mu0) and np.array_equal(fc, fc0) and f == f0, amp
        fresh.close()


@pytest.mark.parametrize("g", [129, 210])  # 8 lanes a cell, and 4
def test_most_cells_of_a_warm_evaluation_take_the_short_path(gpu, g):
    """The bits are the warp kernels' whichever cells they take: that the short
    path takes most of them where little moves, leaves those that move, and
    none in a domain whose squares vanish, shows in the counters alone."""
    p = problems.make(4, g=g, res=200)
    n = p.n
    rng = np.random.default_rng(g)
    s = solver_for(p)
    w = rng.normal(0.0, 0.05 / n, n)
    left = {}
    for amp in (None, 0.0, 0.01, 3.0):
        w = w + (0.0 if amp is None else rng.normal(0.0, amp / n, n))
        s.eval(w)
        c = s.ring_counters()
        assert c["rings_by_warp"] <= n and c["walks_by_warp"] <= n
        left[amp] = c
    assert left[None]["rings_by_warp"] == n  # no ring yet
    assert left[0.0]["rings_by_warp"] + left[0.0]["walks_by_warp"] < n // 4, left
    assert left[0.01]["rings_by_warp"] + left[0.01]["walks_by_warp"] < n // 2, left
    assert left[3.0]["rings_by_warp"] > n // 4, left
    k = 2.0 ** -90
    small = solver_for(problems.SDOTProblem("small", p.xy * k, p.nu * k * k, p.picture, p.size,
                                            np.asarray(p.proj_domain) * k))
    for _ in range(2):
        small.eval(np.zeros(n))
    c = small.ring_counters()
    assert c["rings_by_warp"] < n // 2 and c["walks_by_warp"] == n, c
