"""Certificate walks with many surviving leaves, which are finished by the warp
itself or by a block (k_cells_heavy) as the number of sites has it."""
import numpy as np
import pytest

from caustic_b200 import problems
from test_gpu_parity import check_eval, solver_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gx,gy", [(128, 64), (129, 64)])  # the last size without a limit of leaves, and the next
def test_long_walks_on_both_sides_of_the_limit(gpu, gx, gy):
    rng = np.random.default_rng(gx)
    xy = problems.jittered_grid(rng, gx, gy)
    n = gx * gy
    nu = rng.uniform(0.5, 1.5, n)
    pic = rng.uniform(0.1, 1.0, 96 * 80)
    p = problems.SDOTProblem("walks", xy, nu / nu.sum(), pic / pic.sum(), (96, 80))
    s = solver_for(p)
    # cells far from their sites: every first ring is far too large
    w = 0.1 * np.sin(5.0 * xy[:, 0]) * np.cos(4.0 * xy[:, 1])
    check_eval(p, w, s)
    blocks = s.eval_counters()["walks_by_block"]
    check_eval(p, w + rng.normal(0.0, 1.0 / n, n), s)
    cold = solver_for(p)
    assert np.array_equal(s.eval(w)[1], cold.eval(w)[1])
    assert blocks > 0 or gx == 128
