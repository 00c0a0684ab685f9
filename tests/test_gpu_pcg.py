"""The conjugate-gradient launch of the Newton solve in each of its forms (one
cluster with 1, 2 or 4 rows a thread; a block an SM with 1, 2, 4 or any number
of rows), at sizes that leave the last block part empty."""
import numpy as np
import pytest

from caustic_b200 import capi, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gx,gy", [
    (13, 17),    # one block
    (63, 65),    # 16 blocks of a row a thread
    (65, 64),    # two rows a thread
    (101, 97),   # four rows a thread
    (128, 128),  # the cluster full
    (131, 127),  # the whole GPU, a row a thread
    (211, 203),  # two rows
    (331, 307),  # four rows
    (421, 397),  # any number of rows
])
def test_newton_at_every_form_of_the_linear_solve(gpu, gx, gy):
    n = gx * gy
    rng = np.random.default_rng(n)
    xy = problems.jittered_grid(rng, gx, gy)
    nu = rng.uniform(0.8, 1.2, n)
    res = 256
    px = (np.arange(res) + 0.5) / res
    pic = 1.0 + 0.3 * np.sin(2 * np.pi * px)[:, None] * np.cos(3 * np.pi * px)[None, :]
    with capi.Solver() as s:
        s.set_problem(xy, nu / nu.sum(), pic.ravel() / pic.sum(), (res, res), problems.UNIT_DOMAIN)
        w, st = s.solve_newton(np.zeros(n), tol=1e-6, cg_rtol=1e-3)
        assert st.converged and not st.fallback and st.cg_iterations > 0, st
        _, mu, g, _ = s.eval(w)
        assert (np.abs(g) / (mu - g)).max() <= 1.001e-6
        # a Newton step whose linear system is solved to 1e-3 converges fast
        assert st.newton_iterations <= 12, st
        w2, st2 = s.solve_newton(np.zeros(n), tol=1e-6, cg_rtol=1e-3)
        assert np.array_equal(w, w2) and st2.cg_iterations == st.cg_iterations
