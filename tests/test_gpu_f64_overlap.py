"""The FP64 form's averaged update of overlapped cubes (k = 32, 48, 64) over more
than one tile of 128 state rows and up to nine covers a column, and the columns it
lists for k_overlap_update.

Bar: the FP64 form's 1e-10 against the oracle; repeated runs, and columns beside
listed ones, are bitwise equal.  T' is formed from the members' mean that other
warps use at the same time for the mean increment, so a column's T' and u must not
depend on which warp comes first.
"""
import numpy as np
import pytest

from conftest import field_rel_err, pkg
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.fixture(scope="module")
def letkf():
    pkg("build").build()
    m = pkg("letkf")
    m.load_library()
    return m


@pytest.mark.parametrize("k,nz,cube_n,overlap", [(32, 43, 3, 2), (48, 42, 3, 2), (64, 86, 3, 2), (64, 43, 2, 1)])
def test_row_tiles_and_covers(letkf, k, nz, cube_n, overlap):
    w = pkg("synthetic").small_case(nlat=8, nlon=16, nz=nz, k=k, nobs=400, loc_dist_km=1200.0, seed=k + nz)
    ctx = letkf.LetkfGPU.from_workload(w, cube_n=cube_n, overlap=overlap)
    xa, axa = ctx.run(w.xb, w.axb, w.obs)
    xa_o, axa_o = O.Oracle(w, cube_n=cube_n, overlap=overlap).run()
    assert max(field_rel_err(axa, axa_o, w).values()) <= TOL
    assert max(field_rel_err(xa, xa_o, w).values()) <= TOL
    for _ in range(3):
        xr, ar = ctx.run(w.xb, w.axb, w.obs)
        assert np.array_equal(xr, xa) and np.array_equal(ar, axa)


@pytest.mark.parametrize("k", [32, 64])
def test_listed_columns(letkf, k):
    # a cube with a NaN departure has a NaN transform: the columns it covers are
    # left to k_overlap_update (and NaN), the others are what they are without it
    w = pkg("synthetic").small_case(nlat=9, nlon=18, nz=43, k=k, nobs=400, loc_dist_km=900.0, seed=k)
    ctx = letkf.LetkfGPU.from_workload(w, cube_n=3, overlap=1)
    xa0, axa0 = ctx.run(w.xb, w.axb, w.obs)
    yo = w.obs["yo"].copy()
    yo[17] = np.nan
    xa, axa = ctx.run(w.xb, w.axb, dict(w.obs, yo=yo))
    bad = np.isnan(axa).all(axis=1)
    assert bad.any() and not bad.all()
    assert np.isnan(xa[bad]).all()
    assert np.array_equal(xa[~bad], xa0[~bad]) and np.array_equal(axa[~bad], axa0[~bad])
