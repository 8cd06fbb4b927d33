"""The FP64 vector phases of the iteration: block reductions at every block size, second-order blocks of
the dimensions that have code of their own (2, 3, 4) and of others, and the rule that leaves the dense
pivot test of a second-order block out."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, generators

# the repository's parity tolerance for x on well-posed instances
X_TOL = 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 64, 128, 256])
@pytest.mark.parametrize("soc", [(2,) * 5, (3,) * 5, (4,) * 4, (1, 2, 3, 4, 5, 9), ()])
def test_block_sizes_and_cone_dimensions_against_the_oracle(oracle_mod, threads, soc):
    n = 33 if threads == 32 else 45  # 32 threads: roots of at most 64 rows
    qps = [generators.random_conic_qp(s, n=n, m_zero=3, m_nonneg=20, soc=soc, density=0.3, family=9) for s in range(3)]
    for precision in (0, 1):
        B = BatchSolver(qps, precision=precision, warm_start=0, threads_per_instance=threads)
        x, s, z, infos = B.solve()
        for i, (xi, _, _) in enumerate(B.split(x, s, z)):
            xo, _, _, io, _ = oracle_mod.solve(qps[i], warm_start=0)
            assert infos[i]["status"] == io["status"] == 1
            assert abs(int(infos[i]["iterations"]) - io["iterations"]) <= 1
            assert np.linalg.norm(xi - xo) <= X_TOL * max(1.0, np.linalg.norm(xo))


def pivots_pass(s, z, sreg, deps):
    """The kernel's FP32 bound (socPivotsPass), for rows of s and z."""
    f = np.float32
    s, z = s.astype(f), z.astype(f)
    s0, z0 = s[:, 0], z[:, 0]
    s1, z1 = (np.sqrt(np.sum(v[:, 1:] ** 2, axis=1, dtype=f)) for v in (s, z))
    sm, zm = s0 - s1, z0 - z1
    ok = (sm > f(1e-3) * s0) & (zm > f(1e-3) * z0) & (s0 > f(1e-15)) & (z0 > f(1e-15)) & (s0 < f(1e15)) & (z0 < f(1e15))
    with np.errstate(all="ignore"):
        a, b = np.sqrt(sm * (s0 + s1)), np.sqrt(zm * (z0 + z1))
        t = s0 / a + z0 / b
        hs = (a / b) * t * t
    return ok & (hs * f(1000 * 2.22e-16) < f(0.25) * f(sreg)) & (f(deps) < f(0.25) * f(sreg))


@pytest.mark.parametrize("d", [2, 3, 4, 8])
def test_blocks_that_skip_the_pivot_test_pass_it(d):
    """Over scales of 1e-6 .. 1e6, margins down to 1e-5 of the axis and aligned or random directions:
    a block that the bound lets through has every pivot of -(Hs + 1e-8 I) above 1e-14, with Hs = W W
    formed densely in FP64 in the reference's order."""
    rng = np.random.default_rng(d)
    N = 20000
    u = rng.standard_normal((2, N, d - 1))
    u[1, : N // 2] = -u[0, : N // 2] + 1e-3 * u[1, : N // 2]
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    axis = 10.0 ** rng.uniform(-6, 6, (2, N))
    t = 1.0 - 10.0 ** rng.uniform(-5, 0, (2, N))
    s, z = (np.concatenate([axis[k][:, None], (axis[k] * t[k])[:, None] * u[k]], axis=1) for k in (0, 1))
    sreg, deps = 1e-8, 1e-14
    ok = pivots_pass(s, z, sreg, deps)
    assert 0.02 < ok.mean() < 0.98  # both outcomes are covered
    s, z = s[ok], z[ok]
    flip = np.concatenate([[1.0], -np.ones(d - 1)])
    a, b = (np.sqrt(np.maximum(v[:, 0] ** 2 - np.sum(v[:, 1:] ** 2, axis=1), 1e-12 * v[:, 0] ** 2)) for v in (s, z))
    beta = np.clip(np.sqrt(a / b), 1e-8, 1e8)
    c = np.sqrt(np.maximum((np.sum(s * z, axis=1) / (a * b) + 1.0) / 2.0, 1e-12))
    v = (flip * z / b[:, None] + s / a[:, None]) / (2.0 * c)[:, None]
    v[:, 0] += 1.0
    v /= np.sqrt(2.0 * v[:, :1])
    W = beta[:, None, None] * (2.0 * v[:, :, None] * v[:, None, :] - np.diag(flip))
    Hs = W @ W
    A = -(Hs + sreg * np.eye(d))
    for k in range(d):
        assert np.min(np.abs(A[:, k, k])) > deps
        l = A[:, k + 1:, k] / A[:, k, k][:, None]
        A[:, k + 1:, k + 1:] -= l[:, :, None] * A[:, k, k + 1:][:, None, :]


@pytest.mark.gpu
@pytest.mark.parametrize("contacts,threads", [(1, 32), (10, 32), (11, 64), (21, 64), (22, 128), (42, 128)])
@pytest.mark.parametrize("precision", [0, 1])
def test_wide_blocks_give_the_narrow_blocks_bits(contacts, threads, precision):
    """A batch with an SM for every instance runs 256-thread blocks with the sums of the narrow block:
    the same bits as the narrow block itself, in the solve and in the adjoint."""
    qps = [generators.contact_qp(s, contacts=contacts) for s in range(3)]
    got = []
    for t in (0, threads):
        B = BatchSolver(qps, precision=precision, warm_start=0, threads_per_instance=t, differentiable=1)
        x, s, z, infos = B.solve()
        got.append((x, s, z, infos["iterations"], infos["refine_steps"]) + B.backward(np.ones(B.n_total)))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_wide_blocks_where_a_cta_has_its_sm_alone(precision):
    """More instances than SMs: a bucket whose shared memory leaves one CTA per SM (here 42
    contacts, 120 KB) runs 256-thread blocks, the other bucket (10 contacts) narrow ones; both give the
    bits of the block sizes asked for by hand."""
    qps = [generators.contact_qp(s, contacts=42 if s % 2 else 10) for s in range(320)]
    got = []
    for t in (0, 128, 32):
        B = BatchSolver(qps, precision=precision, warm_start=0, threads_per_instance=t)
        x, s, z, infos = B.solve()
        got.append((B.split(x, s, z), infos["iterations"]))
    for i in range(len(qps)):
        ref = got[1] if i % 2 else got[2]
        assert got[0][1][i] == ref[1][i]
        for a, b in zip(got[0][0][i], ref[0][i]):
            assert np.array_equal(a, b), i
