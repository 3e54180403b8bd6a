"""Sums of the FP64 form's A build at the edges of their fixed point: lists whose
rows or departures differ widely in size and lists that sum coherently.  The tensor-core
path solves them itself; bar against the oracle: 1e-10 of T's and wbar's largest
element."""
import numpy as np
import pytest

from conftest import field_rel_err, pkg
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


@pytest.mark.parametrize("k", [32, 64, 96, 128])
@pytest.mark.parametrize("p,at,strong", [(128, 0, 256), (300, 100, 64), (2000, 0, 64), (2000, 700, 64), (2000, 700, 256),
                                         (2000, 1900, 128)])
def test_strong_rows_side_by_side(letkf, k, p, at, strong):  # noqa: F811
    # consecutive observations 20 times as strong as the others: the 128 that are
    # summed together hold far more than the list's mean
    g = np.random.default_rng(p + at)
    a = 0.05 * g.uniform(0.5, 1.0, p)
    a[at:at + strong] *= 20.0
    hx = _member(k, p, a, k)
    hx[:, 5] = a * g.choice([-1.0, 1.0], p)
    _check(_context(letkf, k), k, hx, np.ones(p, np.float32), g.standard_normal(p), np.ones(p))


@pytest.mark.parametrize("k", [32, 64, 96, 128])
@pytest.mark.parametrize("value", [1.0, 1.96, 1.3370013370013, 0.9999999])
def test_rows_and_departures_that_repeat_a_value(letkf, k, value):  # noqa: F811
    # equal rows have equal digits, whose products line up in every accumulator; the
    # departures' sums pass 2^24 and come back
    g = np.random.default_rng(k)
    p = 777
    hx = np.tile(value * g.choice([-1.0, 1.0, 0.37], (1, k)), (p, 1))
    dep = np.full(p, 1.1 * value)
    _check(_context(letkf, k), k, hx, np.ones(p, np.float32), dep, np.ones(p))
    dep[64:128] *= -0.99
    dep[300:] *= np.where(np.arange(p - 300) // 40 % 2, -1.0, 1.0)
    _check(_context(letkf, k), k, hx, np.ones(p, np.float32), dep, np.ones(p))


@pytest.mark.parametrize("k", [32, 64, 96, 128])
def test_vertical_weights_past_the_first_table(letkf, k):  # noqa: F811
    # lists longer than a table of factors whose strongest rows have next to no
    # vertical weight
    w = pkg("synthetic").small_case(nlat=6, nlon=12, nz=4, k=k, nobs=3000, loc_dist_km=3000.0, seed=k, h_mode=0)
    kw = dict(vert_dist=0.3, cube_nz=2)
    ctx = letkf.LetkfGPU.from_workload(w, h_mode=0, **kw)
    xa, axa = ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (0, 0) and ctx.stats()["max_p"] > 640
    xa_o, axa_o = O.Oracle(w, **kw).run()
    assert max(field_rel_err(axa, axa_o, w).values()) <= TOL
    assert max(field_rel_err(xa, xa_o, w).values()) <= TOL
