"""Bounded waits of the FP64 form's tensor-core kernels that run out (0 polls: at
once): the run returns LETKF_ERR_TIMEOUT, the kernels let their committed products
finish and free their tensor memory, and the next run of the context is bitwise
that of a fresh one."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def letkf():
    pkg("build").build()
    m = pkg("letkf")
    m.load_library()
    return m


@pytest.mark.parametrize("k,kw", [(32, {}), (48, {}), (64, {}), (96, {}), (128, {}), (32, dict(cube_n=3, overlap=1)),
                                  (64, dict(h_mode=0, vert_dist=0.5, cube_nz=2))])
def test_timeout_leaves_context_usable(letkf, k, kw):
    w = pkg("synthetic").small_case(nlat=10, nlon=20, nz=3, k=k, nobs=1200, loc_dist_km=900.0, seed=70 + k,
                                    h_mode=kw.get("h_mode", 1))
    ref = letkf.LetkfGPU.from_workload(w, **kw)
    xa_ref, axa_ref = ref.run(w.xb, w.axb, w.obs)
    ref.close()
    ctx = letkf.LetkfGPU.from_workload(w, **kw)
    for _ in range(2):
        ctx.set_wait_limit(0)
        with pytest.raises(letkf.LetkfError) as ei:
            ctx.run(w.xb, w.axb, w.obs)
        assert ei.value.code == letkf.LETKF_ERR_TIMEOUT
        ctx.set_wait_limit(-1)
        xa, axa = ctx.run(w.xb, w.axb, w.obs)
        assert np.array_equal(xa, xa_ref) and np.array_equal(axa, axa_ref)


@pytest.mark.parametrize("k", [32, 64, 96])
def test_core_batch_reports_the_timeout(letkf, k):
    g = np.random.default_rng(k)
    off = np.array([0, 0, 150, 350], dtype=np.int64)
    t = int(off[-1])
    prob = (off, g.standard_normal((t, k)), np.ones(t, np.float32), g.standard_normal(t), g.uniform(0.1, 1.0, t))
    glat, glon = pkg("synthetic").make_grid(30.0)
    ctx = letkf.LetkfGPU(glat, glon, 1, k, loc_dist_km=500.0, inflation=1.1)
    tr0, w0 = ctx.core_batch(*prob)
    ctx.set_wait_limit(0)
    with pytest.raises(letkf.LetkfError) as ei:
        ctx.core_batch(*prob)
    assert ei.value.code == letkf.LETKF_ERR_TIMEOUT
    ctx.set_wait_limit(-1)
    tr, w = ctx.core_batch(*prob)
    assert np.array_equal(tr, tr0) and np.array_equal(w, w0)
