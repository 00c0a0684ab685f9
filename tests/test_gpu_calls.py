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
