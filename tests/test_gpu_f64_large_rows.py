"""State rows of the FP64 form whose members reach the largest doubles: finite, so the
row is the power-of-two multiple of the ordinary one (T is not observed), bitwise."""
import numpy as np
import pytest

from conftest import pkg
from test_gpu_f64_digits import letkf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [32, 64, 96])
@pytest.mark.parametrize("top", [1.9, 1.97, 1.99999])
def test_largest_doubles(letkf, k, top):  # noqa: F811
    w = pkg("synthetic").small_case(nlat=8, nlon=16, nz=3, k=k, nobs=300, loc_dist_km=1200.0, seed=9)
    keep = w.obs["var"] != 3
    obs = {key: v[keep] for key, v in w.obs.items()}
    ctx = letkf.LetkfGPU.from_workload(w, inflation=0.9)
    t0 = 1 + 2 * w.nz
    xb, axb = w.xb.copy(), w.axb.copy()
    axb[:, t0] = 0.0
    # every column's largest member is `top` with its sign, the others smaller
    big = np.abs(xb[:, t0]).max(axis=1, keepdims=True)
    xb[:, t0] *= top / big
    xa0, axa0 = ctx.run(xb, axb, obs)
    xb[:, t0] = np.ldexp(xb[:, t0], 1023)
    xa, axa = ctx.run(xb, axb, obs)
    assert np.isfinite(xa0).all() and np.abs(xa0[:, t0]).max() < 2.0 and np.abs(axa0[:, t0]).max() < 2.0
    assert np.array_equal(xa[:, t0], np.ldexp(xa0[:, t0], 1023))
    assert np.array_equal(axa[:, t0], np.ldexp(axa0[:, t0], 1023))
