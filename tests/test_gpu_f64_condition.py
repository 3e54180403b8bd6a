"""T and wbar of the FP64 form over the condition number of A', against extended
precision.

Bar: T's error (over its largest element, geometric mean of the seeds) is not above
that of k_core_fp64, an FP64 Jacobi, from 1e3 to 1e6; T's and wbar's errors stay below
eps cond(A') up to 1e8 (an FP64 matrix holds its smallest eigenvalue to that).
"""
import numpy as np
import pytest

from test_gpu_f64_digits import _context, _core_fp64, letkf  # noqa: F401

pytestmark = pytest.mark.gpu
RHO, P = 1.1, 200
LD = np.longdouble


def _problem(k, cond, seed):
    g = np.random.default_rng([k, int(np.log10(cond)), seed])
    hx = g.standard_normal((P, 12)) @ g.standard_normal((12, k)) / 4 + 0.3 * g.standard_normal((P, k))
    hx -= hx.mean(axis=1, keepdims=True)
    rdi = (1.0 / g.uniform(0.5, 2.0, P) ** 2).astype(np.float32)
    rloc, dep = g.uniform(0.01, 1.0, P), g.standard_normal(P)
    y = hx * np.sqrt(rdi * rloc)[:, None]
    return hx * np.sqrt((cond - 1) * (k - 1) / RHO / np.linalg.eigvalsh(y.T @ y)[-1]), rdi, dep, rloc


def _exact(k, hx, rdi, dep, rloc):
    """T and wbar by Newton's method and refinement with extended residuals."""
    s = np.sqrt(rdi.astype(LD) * rloc.astype(LD))
    y = hx.astype(LD) * s[:, None]
    a, g = y.T @ y + LD(k - 1) / LD(RHO) * np.eye(k, dtype=LD), y.T @ (s * dep)
    lam, v = np.linalg.eigh(a.astype(float))
    solve = lambda r: v @ ((v.T @ r.astype(float)) / lam)
    w = solve(g).astype(LD)
    for _ in range(8):
        w = w + solve(g - a @ w).astype(LD)
    root = np.sqrt(lam)
    t = ((v * np.sqrt((k - 1) / lam)) @ v.T).astype(LD)
    for _ in range(6):
        t = (t + t.T) / 2
        r = v.T @ (t @ a @ t / LD(k - 1) - np.eye(k)).astype(float) @ v
        t = t - (np.sqrt(k - 1) * v @ (r / (root[:, None] + root[None, :])) @ v.T).astype(LD)
    return t, w


@pytest.mark.parametrize("k", [32, 48, 64, 96, 128])
def test_errors_against_extended_precision(letkf, k):  # noqa: F811
    assert np.finfo(LD).eps < 1e-18
    seeds = 5 if k <= 64 else 3
    ctx = _context(letkf, k, RHO)
    off = np.arange(seeds + 1, dtype=np.int64) * P
    for cond in (1e1, 1e3, 1e4, 1e5, 1e6, 1e8):
        prob = [_problem(k, cond, s) for s in range(seeds)]
        args = [np.concatenate([p[i] for p in prob]) for i in range(4)]
        tr, w = ctx.core_batch(off, *args)
        if cond <= 1e6:
            assert ctx.general_counts() == (0, 0)
        tr_c, w_c = _core_fp64(letkf, k, RHO, off, *args)
        err = []
        for b in range(seeds):
            t_x, w_x = _exact(k, *prob[b])
            rel = lambda a, x: float(np.abs(a.astype(LD) - x).max() / np.abs(x).max())
            e_t = rel(tr[b].astype(LD) - w[b].astype(LD)[:, None], t_x)
            e_c = rel(tr_c[b].astype(LD) - w_c[b].astype(LD)[:, None], t_x)
            bar = np.finfo(float).eps * cond * (10 if cond < 1e3 else 1)
            assert e_t <= bar and rel(w[b], w_x) <= bar, (cond, b, e_t, rel(w[b], w_x))
            err.append((e_t, e_c))
        e_t, e_c = np.exp(np.log(np.array(err)).mean(axis=0))
        if cond <= 1e6:
            assert e_t <= e_c, (cond, e_t, e_c)
