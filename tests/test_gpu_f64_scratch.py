"""The FP64 form within a limit on its intermediates: smaller blocks of problems give
the same results bitwise; where no block fits, the general kernels solve everything
(1e-10 against the oracle), and the limit can be lifted again."""
import numpy as np
import pytest

from conftest import field_rel_err, pkg
from oracle import oracle as O
from test_gpu_f64_digits import TOL, letkf  # noqa: F401

pytestmark = pytest.mark.gpu


def _bytes(k, n):
    ks = 32 if k <= 32 else 64 if k <= 64 else k
    n *= ks * ks * (12 if k > 64 else 16) + 12 * ks + 16
    if k > 64:
        import torch
        n += 8 * torch.cuda.get_device_properties(0).multi_processor_count * (3 * k * k + k // 4 * 512)
    return n


@pytest.mark.parametrize("k,kw,per_cube", [(32, {}, 1), (64, dict(h_mode=0, vert_dist=0.5, cube_nz=2), 2),
                                           (32, dict(cube_n=2, overlap=1), 1), (96, {}, 1)])
def test_blocks_of_runs(letkf, k, kw, per_cube):  # noqa: F811
    w = pkg("synthetic").small_case(nlat=36, nlon=72, nz=4, k=k, nobs=900, loc_dist_km=900.0, seed=k,
                                    h_mode=kw.get("h_mode", 1))
    ctx = letkf.LetkfGPU.from_workload(w, **kw)
    xa0, axa0 = ctx.run(w.xb, w.axb, w.obs)
    n = w.ncol * per_cube
    for blocks in (1, 2, 3):
        # (a block that does not fit is halved)
        ctx.set_scratch_limit(_bytes(k, max(1200, n // blocks)) + 1)
        for _ in range(2):
            xa, axa = ctx.run(w.xb, w.axb, w.obs)
            assert ctx.general_counts() == (0, 0)
            assert np.array_equal(xa, xa0) and np.array_equal(axa, axa0)
    ctx.set_scratch_limit(1)
    xa, axa = ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts()[0] == n
    assert max(field_rel_err(axa, axa0, w).values()) <= TOL and max(field_rel_err(xa, xa0, w).values()) <= TOL
    ctx.set_scratch_limit(0)
    xa, axa = ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (0, 0)
    assert np.array_equal(xa, xa0) and np.array_equal(axa, axa0)


@pytest.mark.parametrize("k", [32, 48, 64, 96, 128])
def test_no_block_fits(letkf, k):  # noqa: F811
    w = pkg("synthetic").small_case(nlat=8, nlon=16, nz=3, k=k, nobs=300, loc_dist_km=1200.0, seed=k)
    ctx = letkf.LetkfGPU.from_workload(w)
    ctx.set_scratch_limit(1)
    xa, axa = ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (w.ncol, 0)
    xa_o, axa_o = O.Oracle(w).run()
    assert max(field_rel_err(axa, axa_o, w).values()) <= TOL
    assert max(field_rel_err(xa, xa_o, w).values()) <= TOL


def test_more_level_blocks_than_the_smallest_block(letkf):  # noqa: F811
    # one cube's level blocks are one block of problems: it cannot shrink further
    w = pkg("synthetic").small_case(nlat=4, nlon=8, nz=1100, k=32, nobs=200, loc_dist_km=1500.0, seed=1, h_mode=0)
    kw = dict(vert_dist=0.5, cube_nz=1)
    ctx = letkf.LetkfGPU.from_workload(w, **kw)
    xa0, axa0 = ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (0, 0)
    ctx.set_scratch_limit(_bytes(32, 1100) + 1)
    xa, axa = ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (0, 0)
    assert np.array_equal(xa, xa0) and np.array_equal(axa, axa0)
    ctx.set_scratch_limit(_bytes(32, 1099))
    xa, axa = ctx.run(w.xb, w.axb, w.obs)
    assert ctx.general_counts() == (w.ncol * 1100, 0)
    assert max(field_rel_err(xa, xa0, w).values()) <= TOL


@pytest.mark.parametrize("k", [32, 64, 96])
def test_members_without_room_for_the_split_state(letkf, k):  # noqa: F811
    w = pkg("synthetic").small_case(nlat=8, nlon=16, nz=3, k=k, nobs=300, loc_dist_km=1200.0, seed=k)
    xin = w.xb + w.axb[..., None]
    kw = dict(gamma1=0.3, gamma2=0.7, polar_lat_deg=70.0)
    ctx = letkf.LetkfGPU.from_workload(w)
    split = ctx.run_members(xin, w.obs, **kw)
    assert ctx.general_counts() == (0, 0)
    ctx.set_scratch_limit(16 * w.axb.size * (k + 1) - 1)
    fused = ctx.run_members(xin, w.obs, **kw)
    assert ctx.general_counts() == (w.ncol, 0)
    for a, b in zip(fused, split):
        assert max(field_rel_err(a, b, w).values()) <= TOL
