"""Products that the whole-GPU form hands to the other CTAs, against the one-CTA form."""
import numpy as np
import pytest

from conicxx_gb300 import Solver
from test_gpu_products import ragged_qp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,zero,nonneg,soc", [(352, 2, 309, (6, 3)), (352, 2, 310, (6, 3)), (1025, 3, 40, (4, 5))])
def test_first_iteration_of_both_forms(n, zero, nonneg, soc):
    """FP64, sizes of 32 and more slices in a KKT residual and in a product with P alone. Both forms refine their
    KKT solves to a relative residual of 1e-12, so the first iteration's trace (mu, residual norms,
    objectives, steps, tau, kappa) agrees to 1e-12 times the condition of these systems (below 1e3): 1e-9."""
    qp = ragged_qp(5, n, zero, nonneg, soc)
    rows = []
    for whole in (-1, 1):
        S = Solver()
        assert S.setup(qp, precision=0, warm_start=0, whole_gpu_root=whole, record_timings=1)
        assert S.solve().ok()
        rows.append(S.trace()[0])
    assert np.all(np.abs(rows[0][:10] - rows[1][:10]) <= 1e-9 * np.maximum(1.0, np.abs(rows[0][:10])))
