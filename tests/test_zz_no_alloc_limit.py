"""GPU test of the allocation-free batch solve between two sizes: an instance that fits the fixed
working memory but for A's copies in the products' orders works in the batch's own scratch."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, _abi
from conicxx_gb300.problem import QP, Csc

pytestmark = pytest.mark.gpu


def test_noalloc_at_the_fixed_arrays_limit():
    """n = 2816 in FP64: the root's 33.08 MB leave 0.47 MB of the fixed 33.55 MB for the rest; with 5000
    entries of A the working memory is above that, without A's two copies below it. One iteration; the
    results are the device solve's bits (the same kernel on the same inputs)."""
    torch = pytest.importorskip("torch")
    n, m, nnz = 2816, 100, 50
    rng = np.random.default_rng(0)
    rows = np.repeat(np.arange(m), nnz)
    cols = np.concatenate([rng.choice(n, nnz, replace=False) for _ in range(m)])
    P = Csc.from_coo(n, n, np.arange(n), np.arange(n), np.ones(n))
    A = Csc.from_coo(m, n, rows, cols, rng.standard_normal(m * nnz))
    qp = QP(P, rng.standard_normal(n), A, np.ones(m), 0, m, [])
    B = BatchSolver([qp], warm_start=0, precision=_abi.PRECISION_FP64, max_iter=1)
    need = int(B.describe().split("scratchPerCTA=")[1].split()[0])
    cap = ((32 << 20) - 256) // 8
    assert cap < need < cap + 2 * m * nnz, (need, cap)
    stream = torch.cuda.current_stream().cuda_stream
    got = []
    for solve in (B.solve_device, B.solve_device_noalloc):
        out = [torch.full((k,), float("nan"), dtype=torch.float64, device="cuda") for k in (n, m, m)]
        solve(*[t.data_ptr() for t in out], stream)
        torch.cuda.synchronize()
        got.append([t.cpu().numpy() for t in out])
    for a, b in zip(*got):
        assert np.isfinite(a).all() and np.array_equal(a, b)
