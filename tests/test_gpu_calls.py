"""What calls of the C ABI promise besides their values: the memory flag of an
evaluation, cells beyond the largest ring, the memory that a handle holds."""
import ctypes

import numpy as np
import pytest

from caustic_b200 import capi, problems
from test_gpu_parity import solver_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_side", [20, 72])  # results through pinned memory, and straight to the caller's
def test_evaluation_takes_any_other_flag_as_host(gpu, n_side):
    """cot_eval knows device arrays by COT_MEM_DEVICE alone."""
    p = problems.make(1, g=n_side, res=128)
    s = solver_for(p)
    w = np.random.default_rng(1).normal(0.0, 0.1 / p.n, p.n)
    f, mu, g, fc = s.eval(w)
    out = np.empty((3, p.n))
    val = ctypes.c_double()
    rc = s._L.cot_eval(s._h, w.ctypes.data, ctypes.byref(val), out[0].ctypes.data, out[1].ctypes.data,
                       out[2].ctypes.data, 2)
    assert rc == 0 and val.value == f
    assert np.array_equal(out[0], mu) and np.array_equal(out[1], g) and np.array_equal(out[2], fc)


@pytest.mark.parametrize("weighted", [False, True])
def test_centroid_of_a_cell_beyond_the_largest_ring(gpu, weighted):
    """300 neighbours: more vertices than a ring holds.  The cell counts as
    empty, whatever an earlier call found for it."""
    th = 2 * np.pi * np.arange(300) / 300
    # (radii that differ a little, or all the other cells' sides meet in one point)
    r = 0.2 + 1e-6 * np.random.default_rng(0).uniform(-1.0, 1.0, 300)
    xy = np.vstack([[[0.4, 0.45]], np.column_stack([0.4 + r * np.cos(th), 0.45 + r * np.sin(th)])])
    n = len(xy)
    s = capi.Solver()
    s.set_problem(xy, np.ones(n) / n, np.ones(64 * 64) / 4096.0, (64, 64), np.array([0.0, 1.0, 0.0, 1.0]))
    w = np.zeros(n)
    w[0] = 3.0  # the whole domain
    c, ex = s.centroids(w, weighted=weighted)
    assert ex[0] and not ex[1:].any() and np.abs(c[0] - 0.5).max() < 1e-12
    c, ex = s.centroids(np.zeros(n), weighted=weighted)
    assert ex[1:].all() and not ex[0] and np.array_equal(c[0], xy[0])


def test_memory_is_taken_by_the_calls_that_need_it(gpu):
    """A handle that evaluates holds no history, centroids or Anderson vectors;
    a longer history takes the shorter one's place."""
    import torch

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    p = problems.make(4, g=512, res=256)  # 262,144 sites
    w = np.random.default_rng(2).normal(0.0, 0.05 / p.n, p.n)
    warm = solver_for(problems.make(1, g=16, res=32))  # the context, the kernels
    warm.eval(np.zeros(256))
    warm.close()
    n0 = used()
    s = solver_for(p)
    s.eval(w)
    base = used() - n0
    mb = 1 << 20
    # per site: rings 640, neighbour caches 136, vectors and lists 140, the sort
    # 24, its share of a bucket of 16 with its leaf list 22
    assert base <= 980 * p.n + 24 * mb, base / p.n
    s.centroids(w)
    pts = used() - n0 - base
    assert pts <= p.n * 34 + 4 * mb
    for m in (10, 20, 32):
        s.solve(np.zeros(p.n), mode=capi.SOLVE_WOLFE, tol=1e-12, history=m, max_iter=1)
        hist = used() - n0 - base - pts
        assert 16 * m * p.n <= hist <= 16 * m * p.n + 16 * mb, (m, hist / p.n)


def test_a_history_longer_than_the_first_room(gpu):
    """Small problems have room for ten pairs from the start; a longer history
    moves, a shorter one after it stays, and results do not change."""
    p = problems.make(1, g=24, res=96)
    runs = []
    for order in ((10, 24, 10, 3), (3, 10, 24, 10)):
        s = solver_for(p)
        runs.append({m: s.solve(np.zeros(p.n), mode=capi.SOLVE_WOLFE, history=m, max_iter=40, tol=1e-9)[0]
                     for m in order})
    for m in (3, 10, 24):
        assert np.array_equal(runs[0][m], runs[1][m])
