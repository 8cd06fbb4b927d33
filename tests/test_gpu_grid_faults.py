"""A CTA that leaves a whole-GPU launch: every wait is bounded, and no result is formed from work that was
not done. A host-side setting lets one CTA leave before its share of a given job; the waits end after a
short limit and the context stays usable."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, _abi, _lib
from test_gpu_products import ragged_qp

pytestmark = pytest.mark.gpu
WAIT_S = 0.05


def _solve(B, job):
    assert _lib.lib().cxg_batch_grid_fault(B._h, job, WAIT_S) == _abi.OK
    x, _, _, infos = B.solve()
    return int(infos["status"][0]), x, B.backward(np.ones(B.n_total))


@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
def test_no_answer_from_a_job_left_undone(precision):
    """n = 400 and m = 340: factorisations, solves (13 tile rows, so that CTA 1 owns some of them), products on
    the other CTAs (39 slices) and the copy of the root. Whichever job is left undone, the solve reports
    NumericalError and zero gradients; the copy for the adjoint, the last job, is made all the same, so that
    without it and without any fault the solution and the gradients are the same bits."""
    qp = ragged_qp(5, 400, 2, 329, (6, 3))
    B = BatchSolver([qp], precision=precision, warm_start=0, whole_gpu_root=1, differentiable=1)
    ok, x0, g0 = _solve(B, 0)
    assert ok == _abi.STATUS_SOLVED
    lo, hi = 1, 4096  # the first job number that does not come: the smallest that leaves the answer alone, + 1
    while lo < hi:
        mid = (lo + hi) // 2
        if _solve(B, mid)[0] == _abi.STATUS_SOLVED:
            hi = mid
        else:
            lo = mid + 1
    last = lo  # the copy for the adjoint
    assert 60 < last < 4096
    for job in [1, 2, 3] + list(range(last - 14, last)):
        st, _, g = _solve(B, job)
        assert st == _abi.STATUS_NUMERICAL_ERROR, job
        assert all(not v.any() for v in g), job
    for job in (last, last + 1, 0):
        B.update_values(q=qp.q * 2.0)  # another answer in between: the saved root is another one
        _solve(B, 0)
        B.update_values(q=qp.q)
        st, x, g = _solve(B, job)
        assert st == _abi.STATUS_SOLVED and np.array_equal(x, x0)
        for a, b in zip(g, g0):
            assert np.array_equal(a, b), job
