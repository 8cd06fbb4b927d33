"""The allocation-free solve stays within its fixed array: where A's copies in the products' orders would not
fit there for every CTA, the kernel reads A's values through their source indices instead."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, _abi, generators
from conicxx_gb300.problem import QP, Csc

pytestmark = pytest.mark.gpu
CAP = ((32 << 20) - 256) // 8  # doubles of CXG_NOALLOC_SCRATCH_BYTES less the queue counters


def _fields(B):
    return [dict(f.split("=") for f in ln.split() if "=" in f) for ln in B.describe().strip().splitlines()]


def _dense_a(count, n, m, seed):
    """A dense: its copies are a large part of the working memory."""
    out = []
    for i in range(count):
        rng = np.random.default_rng(seed + i)
        A = rng.standard_normal((m, n))
        b = A @ rng.standard_normal(n) * 0.1 + rng.uniform(0.5, 1.5, m)
        out.append(QP(Csc.from_coo(n, n, np.arange(n), np.arange(n), np.ones(n)), rng.standard_normal(n),
                      Csc.from_dense(A, keep_zeros=False), b, 0, m, []))
    return out


def _limit():
    """One instance whose working memory is above the array's size with the copies, below it without: a root
    of 33.08 MB (2816 rows, FP64) and 5000 entries of A."""
    n, m, nnz = 2816, 100, 50
    rng = np.random.default_rng(0)
    cols = np.concatenate([rng.choice(n, nnz, replace=False) for _ in range(m)])
    A = Csc.from_coo(m, n, np.repeat(np.arange(m), nnz), cols, rng.standard_normal(m * nnz))
    return [QP(Csc.from_coo(n, n, np.arange(n), np.arange(n), np.ones(n)), rng.standard_normal(n), A, np.ones(m), 0, m,
               [])]


CASES = {
    "limit": (_limit, 0, 1),
    "config0": (lambda: [generators.config0_qp(700 + i) for i in range(58)], 0, 200),
    "dense": (lambda: _dense_a(96, 60, 400, 3), 1, 200),
    "soc": (lambda: [generators.random_conic_qp(s, n=230, m_zero=5, m_nonneg=40, soc=(3, 4, 6) * 20, density=0.3, family=9)
                     for s in range(100)], 1, 200),
}


@pytest.mark.parametrize("case", CASES)
def test_working_memory_is_the_fixed_arrays(case):
    """Bits of the device solve, in no more memory than the array has; without the copies where it holds no
    CTA with them, or where a CTA takes fewer instances without."""
    torch = pytest.importorskip("torch")
    make, precision, max_iter = CASES[case]
    qps = make()
    B = BatchSolver(qps, warm_start=0, precision=precision, max_iter=max_iter)
    cut = False
    for f in _fields(B):
        need, grid, per = int(f["scratchPerCTA"]), int(f["noallocGrid"]), int(f["noallocPerCTA"])
        assert grid * per <= CAP
        if per < need:
            cut = True
            alone = min(int(f["instances"]), 152)  # one CTA an SM in these cases
            count, copies = int(f["instances"]), min(alone, CAP // need)
            assert grid == min(alone, CAP // per)
            assert copies == 0 or -(-count // grid) < -(-count // copies)
            assert need - per >= 2 * min(qp.A.nnz for qp in qps)
    assert cut, B.describe()
    stream = torch.cuda.current_stream().cuda_stream
    got = []
    for solve in (B.solve_device, B.solve_device_noalloc):
        out = [torch.full((k,), float("nan"), dtype=torch.float64, device="cuda")
               for k in (B.n_total, B.m_total, B.m_total)]
        infos = np.zeros(B.count, dtype=_abi.INFO_DTYPE)
        solve(*[t.data_ptr() for t in out], stream, infos)
        got.append([t.cpu().numpy() for t in out] + [infos["status"], infos["iterations"], infos["refine_steps"]])
    for a, b in zip(*got):
        assert np.isfinite(a).all() and np.array_equal(a, b)
