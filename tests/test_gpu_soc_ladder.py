"""The bound that spares a second-order block its dense pivots, on the device: the level of the regularisation
ladder is the pivots' own, whether the bound is taken or not."""
import numpy as np
import pytest

from conicxx_gb300 import _abi, _lib
from conicxx_gb300._abi import dptr, iptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", range(2, 9))
@pytest.mark.parametrize("sreg", [1e-10, 1e-8, 1e-4])
@pytest.mark.parametrize("deps_of_sreg", [None, 0.2])
def test_the_bound_changes_no_level(d, sreg, deps_of_sreg):
    """Axes of 1e-6 .. 1e6, margins down to 1e-12 of the axis, random and opposed directions; searches from level
    0, 1 and 9; the default pivot limit and one of a fifth of the regularisation (the bound takes a quarter).
    Both answers of the bound occur."""
    rng = np.random.default_rng(d)
    N = 40000
    u = rng.standard_normal((2, N, d - 1))
    u[1, : N // 2] = -u[0, : N // 2] + 1e-3 * u[1, : N // 2]
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    axis = 10.0 ** rng.uniform(-6, 6, (2, N))
    t = 1.0 - 10.0 ** rng.uniform(-12, 0, (2, N))
    s, z = (np.ascontiguousarray(np.concatenate([axis[k][:, None], (axis[k] * t[k])[:, None] * u[k]], axis=1))
            for k in (0, 1))
    deps = 1e-14 if deps_of_sreg is None else deps_of_sreg * sreg
    for start in (0, 1, 9):
        out = np.zeros((N, 3), np.int32)
        assert _lib.lib().cxg_soc_ladder_eval(N, d, dptr(s), dptr(z), sreg, deps, 1e-7, start, iptr(out)) == _abi.OK
        level, exact, spared = out.T
        assert np.array_equal(level, exact)
        assert np.all(level[spared == 1] == start)
        assert 0.002 < spared.mean() < 0.98
