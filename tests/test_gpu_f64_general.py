"""Which problems the FP64 form's tensor-core path solves itself and which it leaves
to the general kernels (letkf_gpu_general_counts): none of ordinary ones, in every
option, and exactly those that do not fit."""
import numpy as np
import pytest

from conftest import pkg
from test_gpu_f64_digits import COUNTS, _context, _problems, letkf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [32, 48, 64, 96, 128])
def test_batched_core(letkf, k):  # noqa: F811
    ctx = _context(letkf, k)
    ctx.core_batch(*_problems(k, COUNTS, 10 + k))
    assert ctx.general_counts() == (0, 0)
    # out of FP32's range, and of the path's
    ctx.core_batch(*_problems(k, [100, 70, 100, 300, 90], 3, np.array([1.0, 1e20, 1.0, 1.0, 1e-20])))
    assert ctx.general_counts() == (1, 0)
    ctx.core_batch(*_problems(k, COUNTS, 10 + k))
    assert ctx.general_counts() == (0, 0)


@pytest.mark.parametrize("k,kw,cubes", [(32, {}, 128), (48, {}, 128), (64, {}, 128), (96, {}, 128), (128, {}, 128),
                                        (32, dict(cube_n=2), 32), (64, dict(h_mode=0, vert_dist=0.5, cube_nz=2), 256),
                                        (96, dict(h_mode=0, vert_dist=0.5, cube_nz=3), 256),
                                        (32, dict(cube_n=3, overlap=1), 32), (64, dict(cube_n=3, overlap=1), 32)])
def test_runs(letkf, k, kw, cubes):  # noqa: F811
    torch = pytest.importorskip("torch")
    w = pkg("synthetic").small_case(nlat=8, nlon=16, nz=4, k=k, nobs=500, loc_dist_km=1200.0, seed=k,
                                    h_mode=kw.get("h_mode", 1))
    ctx = letkf.LetkfGPU.from_workload(w, **kw)
    ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (0, 0)
    # arrays between 16-byte boundaries: everything
    dev = lambda a: torch.zeros(a.size + 1, dtype=torch.float64, device="cuda")[1:].view(a.shape)
    xb, xa = dev(w.xb), dev(w.xb)
    xb.copy_(torch.from_numpy(w.xb))
    axb, axa = torch.from_numpy(w.axb).cuda(), torch.zeros(w.axb.shape, dtype=torch.float64, device="cuda")
    obs = letkf.ObsArrays({key: torch.from_numpy(np.ascontiguousarray(v)).cuda() for key, v in w.obs.items()},
                          device=True)
    torch.cuda.synchronize()
    ctx.run_device(xb, axb, obs, xa, axa)
    torch.cuda.synchronize()
    over = "overlap" in kw
    assert ctx.general_counts() == (0 if over else cubes, w.ncol if over else 0)
    ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (0, 0)


def test_listed_overlap_columns_are_counted(letkf):  # noqa: F811
    w = pkg("synthetic").small_case(nlat=9, nlon=18, nz=3, k=32, nobs=400, loc_dist_km=900.0, seed=32)
    ctx = letkf.LetkfGPU.from_workload(w, cube_n=3, overlap=1)
    yo = w.obs["yo"].copy()
    yo[17] = np.nan
    _, axa = ctx.run(w.xb, w.axb, dict(w.obs, yo=yo))
    problems, columns = ctx.general_counts()
    assert problems > 0 and columns == int(np.isnan(axa).all(axis=1).sum())
