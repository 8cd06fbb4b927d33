"""Row orders and the whole-GPU triangular solve at the edges of their splits.

The sparse products read rows sorted by length, 32 a slice: problems whose rows of P and A have very
different lengths (empty, one entry, dense), and sizes around the slices, against the oracle. The
whole-GPU solve hands row tiles from warp to warp: roots of one tile up to more tiles than the warps of
a CTA, against numpy."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver
from conicxx_gb300.problem import QP, Csc
from test_gpu_dense import quasi_definite
from test_gpu_large import _probe

pytestmark = pytest.mark.gpu
X_TOL = 1e-5  # the repository's parity tolerance for x on well-posed instances


def ragged_qp(seed, n, zero, nonneg, soc):
    """P = diag + one dense row and column + a few entries; A with empty-but-one, short and dense rows."""
    rng = np.random.default_rng(seed)
    m = zero + nonneg + sum(soc)
    M = np.diag(rng.uniform(1.0, 2.0, n))
    M[0, 1:] = M[1:, 0] = 0.1 * rng.standard_normal(n - 1) / np.sqrt(n)
    for _ in range(n):
        i, j = rng.integers(0, n, 2)
        M[i, j] = M[j, i] = M[i, j] + (0.05 if i != j else 0.0) * rng.standard_normal()
    M += np.eye(n) * max(0.0, 0.1 - np.linalg.eigvalsh(M)[0])
    A = np.zeros((m, n))
    for r in range(m):
        k = [1, 1, 2, 3, n][rng.integers(0, 5)]
        A[r, rng.choice(n, size=k, replace=False)] = rng.standard_normal(k)
    x0 = rng.standard_normal(n)
    s0, z0 = np.zeros(m), rng.standard_normal(m)
    s0[zero:zero + nonneg] = rng.uniform(0.5, 1.5, nonneg)
    z0[zero:zero + nonneg] = rng.uniform(0.5, 1.5, nonneg)
    o = zero + nonneg
    for d in soc:
        for v in (s0, z0):
            v[o + 1:o + d] = rng.standard_normal(d - 1)
            v[o] = np.linalg.norm(v[o + 1:o + d]) + rng.uniform(0.5, 1.5)
        o += d
    return QP(Csc.from_dense(np.triu(M), keep_zeros=False), -M @ x0 - A.T @ z0, Csc.from_dense(A, keep_zeros=False),
              A @ x0 + s0, zero, nonneg, list(soc))


@pytest.mark.parametrize("n,zero,nonneg,soc", [(1, 0, 1, ()), (7, 1, 3, (3,)), (31, 0, 33, (2, 5)), (32, 2, 30, ()),
                                               (33, 3, 1, (4,) * 8), (70, 0, 5, (3,) * 3), (97, 5, 128, (6, 3))])
def test_rows_of_every_length_against_the_oracle(oracle_mod, n, zero, nonneg, soc):
    qps = [ragged_qp(s, n, zero, nonneg, soc) for s in range(2)]
    for precision in (0, 1):
        x, _, _, infos = BatchSolver(qps, precision=precision, warm_start=0).solve()
        for i, qp in enumerate(qps):
            xo, _, _, io, _ = oracle_mod.solve(qp, warm_start=0)
            assert infos[i]["status"] == io["status"] == 1
            xi = x[i * n:(i + 1) * n]
            assert np.linalg.norm(xi - xo) <= X_TOL * max(1.0, np.linalg.norm(xo))


# solve tolerance: the factor's of test_gpu_dense (1e-11, 1e-9, 2e-3), cond ~ 1e3, ten-fold for the solve
@pytest.mark.parametrize("arith,tol", [("fp64", 1e-10), ("df64", 1e-8), ("fp32", 2e-2)])
@pytest.mark.parametrize("nr", [1, 32, 33, 128, 129, 255, 257, 300, 545])
def test_grid_solve_at_the_edges_of_its_runs(nr, arith, tol):
    nx = max(1, nr - nr // 8)
    K = quasi_definite(nr, nx, seed=nr)
    b = np.random.default_rng(nr).standard_normal(nr)
    x = _probe(K, nx, b, arith, -1)[2]
    ref = np.linalg.solve(K, b)
    assert np.linalg.norm(x - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("n,zero,nonneg,soc", [(352, 2, 309, (6, 3)), (352, 2, 310, (6, 3)), (1025, 3, 40, (4, 5))])
@pytest.mark.parametrize("precision", [0, 1])
def test_whole_gpu_products_agree_with_one_cta(n, zero, nonneg, soc, precision):
    """The whole-GPU form hands products of more than 32 slices to the other CTAs: 32 and 33 slices in a
    KKT residual, and 33 in a product with P alone, against the one-CTA form."""
    from conicxx_gb300 import Solver

    qp = ragged_qp(5, n, zero, nonneg, soc)
    got = []
    for whole in (-1, 1):
        S = Solver()
        assert S.setup(qp, precision=precision, warm_start=0, whole_gpu_root=whole)
        sol = S.solve()
        assert int(sol.status) == 1
        got.append(np.asarray(sol.x))
    assert np.linalg.norm(got[0] - got[1]) <= X_TOL * max(1.0, np.linalg.norm(got[0]))
