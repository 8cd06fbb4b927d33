"""The adjoint after replaced instances and an allocation-free solve: more size buckets than the last captured
solve had."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, generators
from conicxx_gb300._lib import CxgError

pytestmark = pytest.mark.gpu


def _noalloc(torch, B):
    out = [torch.zeros(k, dtype=torch.float64, device="cuda") for k in (B.n_total, B.m_total, B.m_total)]
    B.solve_device_noalloc(*[t.data_ptr() for t in out], torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()


def test_backward_after_replace_and_an_allocation_free_solve():
    """One bucket becomes four; the gradients are those of a batch made with the new instances."""
    torch = pytest.importorskip("torch")
    qps = [generators.contact_qp(s, contacts=4) for s in range(8)]
    new = [generators.contact_qp(10 + s, contacts=c) for s, c in enumerate((15, 25, 35))]
    B = BatchSolver(qps, warm_start=0, differentiable=1)
    with pytest.raises(CxgError):
        B.backward(np.ones(B.n_total))  # before any solve
    B.solve()
    assert len(B.describe().strip().splitlines()) == 1
    B.replace([1, 3, 6], new)
    assert len(B.describe().strip().splitlines()) == 4
    _noalloc(torch, B)
    got = B.backward(np.ones(B.n_total))
    F = BatchSolver(B.qps, warm_start=0, differentiable=1)
    F.solve()
    for a, b in zip(got, F.backward(np.ones(F.n_total))):
        assert np.array_equal(a, b)
