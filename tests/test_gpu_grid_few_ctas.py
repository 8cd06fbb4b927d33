"""The whole-GPU root on two to four CTAs: the paths of roots with more row tiles than the warps of every SM own
at once (several row tiles a warp in the triangular solves, several runs of tiles a CTA, one warp a tile in the
column phases), at sizes that a test can afford. Every entry takes one order of operations however the work
is spread, so L, D and x are the bits of the launch on every SM."""
import numpy as np
import pytest

from conicxx_gb300 import _abi, _lib
from test_gpu_dense import ARITH, quasi_definite

pytestmark = pytest.mark.gpu
# test_gpu_products' tolerances of the solve
TOL = {"fp64": 1e-10, "df64": 1e-8, "fp32": 2e-2}


def grid_probe(K, nx, b, arith, ctas, linear_solver=_abi.LINSOLVER_QDLDL):
    nr = K.shape[0]
    Kc = np.asfortranarray(K)
    L, D, x = np.zeros((nr, nr), order="F"), np.zeros(nr), np.zeros(nr)
    ns, flags = np.zeros(2, np.int64), np.zeros(3, np.int32)
    rc = _lib.lib().cxg_dense_ldlt_grid(nr, nx, Kc.ctypes.data, b.ctypes.data, ARITH[arith], ctas, linear_solver,
                                        L.ctypes.data, D.ctypes.data, x.ctypes.data, ns.ctypes.data, flags.ctypes.data)
    assert rc == _abi.OK, _lib.lib().cxg_last_error()
    return L, D, x, flags


# row tiles a warp / runs a CTA in the solve, two CTAs. FP64 (four warps): 2/1, 3/1, 4/1, 4/2, 4/3; the other
# two (eight warps): 2/1, 3/1, 4/1, 4/2
@pytest.mark.parametrize("arith,nr", [("fp64", v) for v in (270, 530, 801, 1100, 2100)] +
                         [(a, v) for a in ("df64", "fp32") for v in (530, 1058, 1570, 2100)])
def test_few_ctas_give_the_bits_of_all(arith, nr):
    nx = nr - nr // 8
    K = quasi_definite(nr, nx, seed=nr)
    b = np.random.default_rng(nr).standard_normal(nr)
    ref = grid_probe(K, nx, b, arith, 0)
    assert not ref[3].any()
    xr = np.linalg.solve(K, b)
    assert np.linalg.norm(ref[2] - xr) <= TOL[arith] * np.linalg.norm(xr)
    for ctas in (2, 3, 4):
        got = grid_probe(K, nx, b, arith, ctas)
        assert not got[3].any()
        for g, r in zip(got[:3], ref[:3]):
            assert np.array_equal(g, r), ctas


@pytest.mark.parametrize("arith", ["fp64", "fp32", "df64"])
@pytest.mark.parametrize("pos", [0, 3, 4, 7, 9, 31, 33, 36, 39])
def test_regularized_pivot_in_the_whole_gpu_form(pos, arith):
    """As test_gpu_tiles' test of the one-CTA form: delta = 1e-7 with the row's sign at a zero pivot, every other
    pivot exactly what it is."""
    d = np.arange(1.0, 41.0)
    d[36:] *= -1.0
    d[pos] = 0.0
    _, D, _, flags = grid_probe(np.diag(d), 36, np.ones(40), arith, 0, _abi.LINSOLVER_REGULARIZED)
    assert not flags.any()
    assert D[pos] == pytest.approx(1e-7 if pos < 36 else -1e-7, rel=1e-6)
    assert np.array_equal(np.delete(D, pos), np.delete(d, pos))


def test_more_ctas_than_the_device_holds_are_refused():
    K, b = np.eye(4), np.ones(4)
    out = np.zeros(16)
    for ctas, rc in ((1, _abi.E_INVALID), (-1, _abi.E_INVALID), (100000, _abi.E_CUDA)):
        assert _lib.lib().cxg_dense_ldlt_grid(4, 4, K.ctypes.data, b.ctypes.data, 0, ctas, 0, out.ctypes.data, None,
                                              None, None, None) == rc
