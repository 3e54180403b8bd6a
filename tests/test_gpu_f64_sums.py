"""Sums of the FP64 form's A build at the edges of their fixed point: lists whose
rows or departures differ widely in size and lists that sum coherently.  The tensor-core
path solves them itself; bar against the oracle: 1e-10 of T's and wbar's largest
element."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_f64_digits import TOL, _context, letkf  # noqa: F401

pytestmark = pytest.mark.gpu


def _check(ctx, k, hx, rdi, dep, rloc):
    tr, w = ctx.core_batch(np.array([0, hx.shape[0]]), hx, rdi, dep, rloc)
    assert ctx.general_counts() == (0, 0)
    t_o, w_o = O.letkf_core(hx, rdi, dep, rloc, 1.1)
    assert np.max(np.abs(w[0] - w_o)) <= TOL * np.abs(w_o).max()
    assert np.max(np.abs((tr[0] - w[0][:, None]) - (t_o - w_o[:, None]))) <= TOL * np.abs(t_o - w_o[:, None]).max()


def _member(k, p, a, seed):
    """Rows with one coherent member a and small noise in the others."""
    g = np.random.default_rng(seed)
    hx = 0.02 * a[:, None] * g.standard_normal((p, k))
    hx[:, 3] = a
    return hx


@pytest.mark.parametrize("k", [32, 64, 96, 128])
@pytest.mark.parametrize("p,weak", [(700, 0.05), (4000, 0.02), (10000, 0.01), (30000, 0.005)])
def test_one_strong_row_among_coherent_weak_ones(letkf, k, p, weak):  # noqa: F811
    # sum |y| over the largest |y| is far above sum y^2 over its square, and every
    # departure is about as large as the largest: g is near its bound and A far
    # from its own.  Just below a power of two the integers are at their largest
    g = np.random.default_rng(p)
    a = 1.96 * weak * g.uniform(0.9, 1.0, p)
    a[p // 3] = 1.96
    _check(_context(letkf, k), k, _member(k, p, a, k), np.ones(p, np.float32), g.uniform(1.7, 1.96, p), np.ones(p))
