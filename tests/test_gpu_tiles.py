"""GPU tests of the root factor's tile operations at the edges of their splits: sizes around the
8-row leaf blocks and the 32-row tiles, every number of warps that splits the work differently.

However the work is spread, every entry takes one order of operations, so L and D are the same bits
for every block size; and they agree with numpy's LDL' within test_gpu_dense's tolerances."""
import numpy as np
import pytest

from conicxx_gb300 import _abi
from test_gpu_dense import TOL, ldlt_ref, probe, quasi_definite

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ["fp64", "fp32", "df64"])
@pytest.mark.parametrize("nr", [1, 7, 8, 9, 24, 25, 31, 33, 41, 65, 96, 129, 161, 190])
def test_factor_is_the_same_for_every_split(nr, arith):
    nx = max(1, nr - nr // 8)
    K = quasi_definite(nr, nx, seed=nr)
    b = np.random.default_rng(nr).standard_normal(nr)
    ref = None
    # 32 .. 256 threads: one warp; two; an odd number; four; more than four; eight
    for threads in (32, 64, 96, 128, 160, 256):
        L, D, x, _, flags = probe(K, nx, b, arith, threads)
        assert flags[0] == 0 and flags[1] == 0
        if ref is None:
            ref = (L, D)
            L0, D0 = ldlt_ref(K)
            tol = TOL[arith]
            assert np.max(np.abs(D - D0)) <= tol * np.max(np.abs(D0))
            assert np.max(np.abs(L - L0)) <= tol * max(1.0, np.max(np.abs(L0)))
        assert np.array_equal(L, ref[0]) and np.array_equal(D, ref[1]), threads


@pytest.mark.parametrize("arith", ["fp64", "df64"])
@pytest.mark.parametrize("nr", [64, 65, 97, 545, 577, 801])
def test_whole_gpu_update_tile_by_tile(nr, arith):
    """The whole-GPU trailing update at its edges: no tile beside the lookahead's (2 tile columns),
    two (3), then fewer tiles than CTAs, about one each (18 tile columns: 152 tiles in the first
    step), and more than one each (both copy buffers in turn)."""
    nx = nr - nr // 8
    K = quasi_definite(nr, nx, seed=nr)
    b = np.random.default_rng(nr).standard_normal(nr)
    L, D, x, _, flags = probe(K, nx, b, arith, -1)
    assert flags[0] == 0 and flags[1] == 0
    L0, D0 = ldlt_ref(K)
    tol = TOL[arith]
    assert np.max(np.abs(D - D0)) <= tol * np.max(np.abs(D0))
    assert np.max(np.abs(L - L0)) <= tol * max(1.0, np.max(np.abs(L0)))


@pytest.mark.parametrize("arith", ["fp64", "fp32", "df64"])
@pytest.mark.parametrize("pos", [0, 3, 4, 7, 9, 31, 33, 36, 39])
def test_regularized_pivot_at_every_place_of_a_leaf(pos, arith):
    """A zero pivot at the edges of the leaf's two halves, in the last block and among the Zero-cone rows:
    the rule puts delta = 1e-7 with the row's sign there; every other pivot stays exactly what it is."""
    d = np.arange(1.0, 41.0)
    d[36:] *= -1.0
    d[pos] = 0.0
    _, D, _, _, flags = probe(np.diag(d), 36, np.ones(40), arith, linear_solver=_abi.LINSOLVER_REGULARIZED)
    assert flags[0] == 0
    assert D[pos] == pytest.approx(1e-7 if pos < 36 else -1e-7, rel=1e-6)
    assert np.array_equal(np.delete(D, pos), np.delete(d, pos))
