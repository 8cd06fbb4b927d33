"""Sizes at the edge of a CTA's shared memory: second-order blocks take eight doubles of it each."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, _abi, _lib
from conicxx_gb300._abi import dptr, iptr
from conicxx_gb300.problem import QP, Csc

pytestmark = pytest.mark.gpu


def test_cone_sets_up_to_200_kb():
    """2560 second-order blocks of one row: 2 * 2560 + 8 * 2560 doubles are 200 KB, the most that the cone
    evaluation takes; one block more is refused. On blocks of one row W = sqrt(s / z), within a few
    roundings (two square roots, two divisions and a product: 1e-14)."""
    rng = np.random.default_rng(0)
    for k, rc in ((2560, _abi.OK), (2561, _abi.E_UNSUPPORTED)):
        s, z, u = (rng.uniform(0.5, 2.0, k) for _ in range(3))
        out, dims = np.zeros(k), np.ones(k, np.int32)
        assert _lib.lib().cxg_cones_eval(0, 0, 0, k, iptr(dims), dptr(s), dptr(z), dptr(u), None, 0.0, dptr(out), None,
                                         None) == rc
        if rc == _abi.OK:
            assert np.max(np.abs(out - np.sqrt(s / z) * u)) < 1e-14 * 4


def test_root_beside_many_second_order_blocks_stays_in_shared_memory():
    """n = 160 and 210 blocks of three rows: reductions 1280 bytes, vectors (10 n + 15 m + 160 + 8 * 210) * 8,
    the FP64 root 15 tiles of 8448: 231,120 of the 231,424 bytes that a CTA may lay out."""
    n, k = 160, 210
    rng = np.random.default_rng(1)
    rows = np.arange(3 * k)
    A = Csc.from_coo(3 * k, n, rows, rng.integers(0, n, 3 * k), rng.standard_normal(3 * k))
    P = Csc.from_coo(n, n, np.arange(n), np.arange(n), np.ones(n))
    b = np.zeros(3 * k)
    b[::3] = 2.0
    qp = QP(P, rng.standard_normal(n), A, b, 0, 0, [3] * k)
    B = BatchSolver([qp], precision=_abi.PRECISION_FP64, warm_start=0)
    assert "vecInSmem=1 rootInSmem=1 root64InSmem=1" in B.describe(), B.describe()
    assert B.solve()[3]["status"][0] == _abi.STATUS_SOLVED
