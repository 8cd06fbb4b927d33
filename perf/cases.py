"""The work that a program has this library do, as timed cases: single problems through `Solver`
(ConicXX's own per-problem call), batches of friction-contact problems through `BatchSolver` (one
simulation timestep), and the differentiable layer `QPLayer` (forward, and forward + backward).

Sizes are those of the library's generators, tests and benchmark. Every input is a function of the
case and the seed alone."""
import math

import numpy as np
import torch

from conicxx_gb300 import BatchSolver, Solver
from conicxx_gb300.problem import QP, Csc, sym_upper_matvec
from conicxx_gb300.torch_layer import QPLayer

MIXED, FP64 = "mixed", "fp64"
PRECISION = {FP64: 0, MIXED: 1}


# ---- cases ---------------------------------------------------------------------------------
def listed():
    return [
        # a controller's few-variable problem, re-solved with new linear terms: latency of one call
        dict(name="solver_n12", kind="sparse", n=12, precision=FP64),
        # a mid-size problem in mixed precision through the same call
        dict(name="solver_n90_mixed", kind="sparse", n=90, precision=MIXED),
        # the 200-variable, 300-row random conic QP, at the call's default precision
        dict(name="solver_n200", kind="sparse", n=200, precision=FP64),
        # one problem whose root is spread over the whole GPU: the smallest such sizes, FP64 ...
        dict(name="solver_lasso_g60", kind="lasso", groups=60, precision=FP64),
        # ... mixed precision, a sparse QP of 1000 variables ...
        dict(name="solver_sparse_n1000", kind="large", n=1000, precision=MIXED),
        # ... and one large enough for the paired tile columns of the factor
        dict(name="solver_sparse_n5400", kind="large", n=5400, precision=MIXED),
        # the contacts of one small scene, timestep after timestep from host arrays
        dict(name="contact_step_24", kind="step", count=24, cmin=4, cmax=24, precision=MIXED),
        # a few hundred scenes in FP64, data on the device
        dict(name="contact_192_fp64", kind="contact", count=192, cmin=4, cmax=64, precision=FP64),
        # a few hundred scenes in mixed precision
        dict(name="contact_512", kind="contact", count=512, cmin=4, cmax=64, precision=MIXED),
        # the benchmark's batch: 4096 contact problems of 4 to 64 contacts
        dict(name="contact_4096", kind="contact", count=4096, cmin=4, cmax=64, precision=MIXED),
        # the layer's evaluation pass: 1024 problems of 100 variables and 150 rows
        dict(name="layer_forward_1024", kind="layer", count=1024, n=100, train=False),
        # one training step of the layer: forward, loss, gradients of every problem value
        dict(name="layer_train_128", kind="layer", count=128, n=100, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sparse", "sparse", "lasso", "large", "step", "contact", "contact", "layer"])
    precision = rng.choice([MIXED, FP64])
    if kind == "sparse":
        return dict(kind=kind, n=_log(rng, 8, 230), precision=precision)
    if kind == "lasso":
        return dict(kind=kind, groups=_log(rng, 32, 120), precision=precision)
    if kind == "large":
        return dict(kind=kind, n=_log(rng, 600, 4800 if precision == MIXED else 1500), precision=precision)
    if kind == "step":
        return dict(kind=kind, count=_log(rng, 1, 64), cmin=4, cmax=rng.randint(8, 64), precision=precision)
    if kind == "contact":
        cmin = rng.randint(1, 16)
        return dict(kind=kind, count=_log(rng, 32, 1500), cmin=cmin, cmax=rng.randint(cmin + 8, 64),
                    precision=precision)
    return dict(kind=kind, count=_log(rng, 8, 800), n=rng.randint(40, 120), train=rng.random() < 0.5)


# ---- problems ------------------------------------------------------------------------------
def _gen(*key):
    return np.random.Generator(np.random.PCG64(np.random.SeedSequence([int(k) & 0xFFFFFFFF for k in key])))


def _upper(M, pattern):
    """Upper triangle of the symmetric M on a symmetric boolean pattern (diagonal kept), in CSC."""
    n = M.shape[0]
    c, r = np.nonzero(np.tril(pattern | np.eye(n, dtype=bool)))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(c, minlength=n))])
    return Csc((n, n), ptr.astype(np.int32), r.astype(np.int32), M[r, c])


def _csc(M, mask):
    c, r = np.nonzero(mask.T)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(c, minlength=M.shape[1]))])
    return Csc(M.shape, ptr.astype(np.int32), r.astype(np.int32), M[r, c])


def _interior(rng, zero, nonneg, soc, dual):
    parts = [rng.standard_normal(zero) if dual else np.zeros(zero), rng.uniform(0.5, 1.5, nonneg)]
    for d in soc:
        u = rng.standard_normal(d - 1)
        parts.append(np.concatenate([[np.linalg.norm(u) + rng.uniform(0.5, 1.5)], u]))
    return np.concatenate(parts)


def _random_qp(rng, n, zero, nonneg, soc, density, pattern=None):
    """A random conic QP with a strictly feasible primal-dual pair (generators.random_conic_qp);
    `pattern` (default rng) draws the sparsity patterns, rng the values."""
    pattern = pattern or rng
    m = zero + nonneg + sum(soc)
    hit = pattern.random((n, n)) < density
    mask = pattern.random((m, n)) < density
    empty = np.flatnonzero(~mask.any(axis=1))
    mask[empty, pattern.integers(0, n, empty.size)] = True
    M = np.where(hit, rng.standard_normal((n, n)), 0.0)
    hit = hit.astype(np.float32)
    P = _upper(M.T @ M + 1e-2 * np.eye(n), (hit.T @ hit) > 0.5)
    Ad = np.where(mask, rng.standard_normal((m, n)), 0.0)
    x0 = rng.standard_normal(n)
    s0, z0 = _interior(rng, zero, nonneg, soc, False), _interior(rng, zero, nonneg, soc, True)
    return QP(P=P, q=-sym_upper_matvec(P, x0) - Ad.T @ z0, A=_csc(Ad, mask), b=Ad @ x0 + s0, zero=zero, nonneg=nonneg,
              soc=list(soc))


def _sparse(case, seed):
    """n variables with the constraint mix of the 200-variable benchmark problem, scaled."""
    n = case["n"]
    zero, nonneg, nsoc = n // 10, max(1, (4 * n) // 5), max(1, n // 5)
    return _random_qp(_gen(10, seed, n), n, zero, nonneg, [3] * nsoc, max(0.05, min(0.5, 4.0 / n)))


def _layer_qp(seed, i, n):
    # a layer's patterns are fixed, its values come with each batch
    return _random_qp(_gen(13, seed, i), n, n // 10, n, [4] * (n // 10), 0.05, pattern=_gen(15, i, n))


def _contact(rng, c):
    """One friction-contact problem as generators.contact_qp builds them: c contacts, each on two
    of ceil(c/4) bodies, P = J Minv J' + 1e-6 I, cones R^c_+ x c Q^3."""
    n, k = 3 * c, (c + 3) // 4
    J = np.zeros((c, 3, k, 6))
    ar = np.arange(c)
    first = rng.integers(0, k, c)
    J[ar, :, first] = rng.standard_normal((c, 3, 6))
    touch = np.zeros((c, k), dtype=bool)
    touch[ar, first] = True
    if k >= 2:
        second = (first + 1 + rng.integers(0, k - 1, c)) % k
        J[ar, :, second] = rng.standard_normal((c, 3, 6))
        touch[ar, second] = True
    G = rng.standard_normal((k, 6, 6))
    Minv = G @ G.transpose(0, 2, 1) / 6.0 + 0.5 * np.eye(6)
    JM = np.einsum("nkb,kbd->nkd", J.reshape(n, k, 6), Minv).reshape(n, 6 * k)
    touch = touch.astype(np.float32)
    share = np.repeat(np.repeat((touch @ touch.T) > 0.5, 3, axis=0), 3, axis=1)
    P = _upper(JM @ J.reshape(n, 6 * k).T + 1e-6 * np.eye(n), share)
    q = 0.1 * rng.standard_normal(n)
    mu = rng.uniform(0.2, 1.0, c)
    # column 3 i: the normal force (its own row, then -mu in the cone); 3 i + 1, 3 i + 2: friction
    rows = np.stack([ar, c + 3 * ar, c + 3 * ar + 1, c + 3 * ar + 2], axis=1).ravel()
    vals = np.stack([-np.ones(c), -mu, -np.ones(c), -np.ones(c)], axis=1).ravel()
    ptr = np.concatenate([[0], np.cumsum(np.tile([2, 1, 1], c))])
    A = Csc((4 * c, n), ptr.astype(np.int32), rows.astype(np.int32), vals)
    return QP(P=P, q=q, A=A, b=np.zeros(4 * c), zero=0, nonneg=c, soc=[3] * c)


def _large(case, seed):
    """generators.large_sparse_qp at n variables (zero, nonneg and cone rows in its proportions)."""
    from conicxx_gb300 import generators

    n = case["n"]
    return generators.large_sparse_qp(seed, n=n, m_zero=n // 10, m_nonneg=(6 * n) // 5, n_soc=n // 10)


def _lasso(case, seed):
    from conicxx_gb300 import generators

    return generators.group_lasso_socp(seed, groups=case["groups"])


def _problems(case, seed):
    kind = case["kind"]
    if kind in ("sparse", "large", "lasso"):
        return [{"sparse": _sparse, "large": _large, "lasso": _lasso}[kind](case, seed)]
    if kind == "layer":
        return [_layer_qp(seed, i, case["n"]) for i in range(case["count"])]
    # contacts per problem ~ U{cmin..cmax}, the same for every seed: outputs keep their sizes
    contacts = _gen(12, case["count"], case["cmin"], case["cmax"]).integers(case["cmin"], case["cmax"] + 1, case["count"])
    return [_contact(_gen(11, seed, i), int(c)) for i, c in enumerate(contacts)]


# ---- one pass ------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    qps = _problems(case, seed)
    if kind in ("sparse", "large", "lasso"):
        solver = Solver()
        assert solver.setup(qps[0], precision=PRECISION[case["precision"]], warm_start=0)
        return dict(kind=kind, solver=solver, q=qps[0].q)
    if kind == "step":
        batch = BatchSolver(qps, precision=PRECISION[case["precision"]], warm_start=0)
        return dict(kind=kind, batch=batch, values=batch.concat_values())
    if kind == "contact":
        batch = BatchSolver(qps, precision=PRECISION[case["precision"]], warm_start=0)
        out = [torch.empty(k, dtype=torch.float64, device="cuda") for k in (batch.n_total, batch.m_total, batch.m_total)]
        return dict(kind=kind, batch=batch, out=out)
    layer = QPLayer(qps)
    values = [torch.from_numpy(v).cuda().requires_grad_(case["train"]) for v in layer.solver.concat_values()]
    target = torch.from_numpy(_gen(14, seed).standard_normal(layer.solver.n_total)).cuda()
    return dict(kind=kind, layer=layer, values=values, target=target, train=case["train"])


def run(state):
    kind = state["kind"]
    if kind in ("sparse", "large", "lasso"):
        # the per-timestep loop of the C++ API: new values, solve, read the solution
        assert state["solver"].update_data(q=state["q"])
        sol = state["solver"].solve()
        return dict(x=sol.x, s=sol.s, z=sol.z, status=int(sol.status), iterations=int(sol.info["iterations"]))
    if kind == "step":
        state["batch"].update_values(*state["values"])
        x, s, z, infos = state["batch"].solve()
        return dict(x=x, s=s, z=z, status=infos["status"], iterations=infos["iterations"])
    if kind == "contact":
        x, s, z = state["out"]
        state["batch"].solve_device(x.data_ptr(), s.data_ptr(), z.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return dict(x=x, s=s, z=z)
    if not state["train"]:
        with torch.no_grad():
            return dict(x=state["layer"](*state["values"]))
    x = state["layer"](*state["values"])
    loss = 0.5 * (x - state["target"]).square().sum()
    grads = torch.autograd.grad(loss, state["values"])
    return dict(x=x.detach(), P=grads[0], q=grads[1], A=grads[2], b=grads[3])


# ---- what a pass cannot do without ---------------------------------------------------------
_ITERATIONS = 12  # interior-point iterations of an ordinary problem of these families


def _shape(case):
    """(problems, variables, rows, root rows, nonzeros of P's upper triangle, of A) on average."""
    kind = case["kind"]
    if kind == "sparse":
        n = case["n"]
        m = n // 10 + max(1, (4 * n) // 5) + 3 * max(1, n // 5)
        d = max(0.05, min(0.5, 4.0 / n))
        return 1, n, m, n + n // 10, 0.5 * n * n * (1 - (1 - d * d) ** n), m * n * d
    if kind == "large":
        n = case["n"]
        m = n // 10 + (6 * n) // 5 + 2 * (n // 10)
        return 1, n, m, n + n // 10, 6 * n, 8 * m
    if kind == "lasso":
        g = case["groups"]
        return 1, 17 * g, 17 * g, 17 * g, 20 * g * 72, 17 * g
    if kind == "layer":
        n = case["n"]
        m = n // 10 + n + 4 * (n // 10)
        return case["count"], n, m, n + n // 10, 0.5 * n * n * (1 - (1 - 0.0025) ** n), 0.05 * m * n
    c = 0.5 * (case["cmin"] + case["cmax"])
    return case["count"], 3 * c, 4 * c, 3 * c, 0.5 * 9 * c * min(c, 15.0), 4 * c


def work(case):
    count, n, m, nr, nnz_p, nnz_a = _shape(case)
    train = case.get("train", False)
    values = nnz_p + nnz_a + n + m
    per_iteration = nr ** 3 / 3 + 6 * nr ** 2 + 12 * (2 * nnz_p + nnz_a)
    return {"bytes": count * 8 * (values * (3 if train else 1) + n + 2 * m),
            "flops": count * (_ITERATIONS * per_iteration + (2 * nr ** 2 if train else 0))}


# ---- the same solutions in plain numpy -----------------------------------------------------
def _dense(qp):
    n, m = qp.n, qp.m
    U = np.zeros((n, n))
    U[qp.P.indices, qp.P.col_of_entries()] = qp.P.data
    A = np.zeros((m, n))
    A[qp.A.indices, qp.A.col_of_entries()] = qp.A.data
    return U + U.T - np.diag(np.diag(U)), A


def _soc_unit(v):
    """sqrt(v0^2 - |v1|^2) of the rows of v, without cancellation."""
    t = np.linalg.norm(v[:, 1:], axis=1)
    return np.sqrt(np.maximum((v[:, 0] - t) * (v[:, 0] + t), 1e-300))


def _optimum(qp):
    """(x, s) of a conic QP whose second-order blocks have one dimension, by a dense primal-dual
    interior-point method with Nesterov-Todd scaling, run until it makes no more progress."""
    P, A = _dense(qp)
    q, b, n, m, p, l = qp.q, qp.b, qp.n, qp.m, qp.zero, qp.nonneg
    nb = len(qp.soc)
    d = qp.soc[0] if nb else 1
    blocks = lambda v: v[p + l:].reshape(nb, d)  # noqa: E731
    flip = np.concatenate([[1.0], -np.ones(d - 1)])
    e = np.zeros(m)
    e[p:p + l] = 1.0
    e[p + l::d] = 1.0 if nb else 0.0
    degree = l + nb
    x, s, z = np.zeros(n), e.copy(), e.copy()

    def product(u, v):
        out = np.zeros(m)
        out[p:p + l] = u[p:p + l] * v[p:p + l]
        U, V = blocks(u), blocks(v)
        blocks(out)[:] = U[:, :1] * V + V[:, :1] * U
        blocks(out)[:, 0] = (U * V).sum(axis=1)
        return out

    def divide(u, w):
        out = np.zeros(m)
        out[p:p + l] = w[p:p + l] / u[p:p + l]
        U, W = blocks(u), blocks(w)
        det = _soc_unit(U)[:, None] ** 2
        nu = (U[:, 1:] * W[:, 1:]).sum(axis=1, keepdims=True)
        blocks(out)[:, 1:] = ((nu / U[:, :1] - W[:, :1]) * U[:, 1:] + det / U[:, :1] * W[:, 1:]) / det
        blocks(out)[:, :1] = (U[:, :1] * W[:, :1] - nu) / det
        return out

    def longest(v, dv):
        t = 1.0
        neg = dv[p:p + l] < 0
        if neg.any():
            t = min(t, float(np.min(-v[p:p + l][neg] / dv[p:p + l][neg])))
        V, D = blocks(v), blocks(dv)
        a = D[:, 0] ** 2 - (D[:, 1:] ** 2).sum(axis=1)
        h = V[:, 0] * D[:, 0] - (V[:, 1:] * D[:, 1:]).sum(axis=1)
        c = _soc_unit(V) ** 2
        root = np.sqrt(np.maximum(h * h - a * c, 0.0))
        with np.errstate(divide="ignore", invalid="ignore"):
            far = np.where(h < 0, np.where(h * h >= a * c, c / (-h + root), np.inf),
                           np.where(a < 0, (-h - root) / a, np.inf))
        return min(t, float(np.min(far))) if nb else t

    best, kept, idle = math.inf, (x, s), 0
    for _ in range(60):
        rd, rp = P @ x + A.T @ z + q, A @ x + s - b
        mu = float(s @ z) / max(degree, 1)
        err = max(np.max(np.abs(rd)), np.max(np.abs(rp)), degree * mu)
        idle = 0 if err < best else idle + 1
        if idle > 4:
            break
        if idle == 0:
            best, kept = err, (x, s)
        # scaling W = diag(sqrt(s/z)) on R_+, beta (2 v v' - J) on each cone
        w = np.sqrt(s[p:p + l] / z[p:p + l])
        S, Z = blocks(s), blocks(z)
        sa, zb = _soc_unit(S), _soc_unit(Z)
        beta = np.sqrt(sa / zb)
        sn, zn = S / sa[:, None], Z / zb[:, None]
        gam = np.sqrt(0.5 * (1.0 + (sn * zn).sum(axis=1)))
        v = (sn + flip * zn) / (2.0 * gam)[:, None]
        v[:, 0] += 1.0
        v /= np.sqrt(2.0 * v[:, :1])

        def apply(u, inverse=False):
            out = np.zeros(m)
            out[p:p + l] = u[p:p + l] / w if inverse else u[p:p + l] * w
            U, vv = blocks(u), (v * flip if inverse else v)
            t = 2.0 * vv * (vv * U).sum(axis=1, keepdims=True) - flip * U
            blocks(out)[:] = t / beta[:, None] if inverse else t * beta[:, None]
            return out

        K = np.zeros((n + m, n + m))
        K[:n, :n], K[:n, n:], K[n:, :n] = P, A.T, A
        K[n + p + np.arange(l), n + p + np.arange(l)] = -w * w
        J = np.diag(flip)
        for i in range(nb):
            W = beta[i] * (2.0 * np.outer(v[i], v[i]) - J)
            o = n + p + l + i * d
            K[o:o + d, o:o + d] = -W @ W
        try:
            inv = np.linalg.inv(K)
        except np.linalg.LinAlgError:
            break
        lam = apply(z)

        def direction(comp):
            rhs = np.concatenate([-rd, -rp - apply(divide(lam, comp))])
            t = inv @ rhs
            t = t + inv @ (rhs - K @ t)
            dz = t[n:]
            ds = apply(divide(lam, comp)) - apply(apply(dz))
            ds[:p] = 0.0
            return t[:n], ds, dz

        dx, ds, dz = direction(-product(lam, lam))
        t = min(longest(s, ds), longest(z, dz))
        sigma = (1.0 - t) ** 3
        dx, ds, dz = direction(-product(lam, lam) - product(apply(ds, True), apply(dz)) + sigma * mu * e)
        t = 0.99 * min(longest(s, ds), longest(z, dz))
        x, s, z = x + t * dx, s + t * ds, z + t * dz
        if not (np.isfinite(x).all() and np.isfinite(s).all() and np.isfinite(z).all()):
            break
    return kept


def exact(case, seed):
    # dense solves on the host: a single problem of up to 230 variables, or a few dozen contacts
    kind = case["kind"]
    if kind not in ("sparse", "step") or case.get("count", 1) * case.get("cmax", 1) > 64 * 24:
        return None
    with np.errstate(all="ignore"):
        got = [_optimum(qp) for qp in _problems(case, seed)]
    # the multipliers of these problems are not unique; counts and states have no 64-bit value
    return dict(x=np.concatenate([g[0] for g in got]), s=np.concatenate([g[1] for g in got]), z=None, status=None,
                iterations=None)
