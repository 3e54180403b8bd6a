"""A captured FP64 run after other calls on its context: the batched core with more
problems and rows than the run has leaves every buffer of the graph where it was, so
a replay is bitwise the separate run (k = 64 mixed: likewise)."""
import numpy as np
import pytest

from conftest import pkg
from test_gpu_batch import _device_case, letkf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,prec", [(32, 0), (64, 0), (96, 0), (16, 0), (64, 1)])
def test_replay_after_core_batch(letkf, k, prec):  # noqa: F811
    torch = pytest.importorskip("torch")
    w = pkg("synthetic").small_case(nlat=8, nlon=16, nz=3, k=k, nobs=300, loc_dist_km=900.0, seed=k)
    ctx = letkf.LetkfGPU.from_workload(w, precision=prec)
    b = _device_case(letkf, torch, w)
    batch = letkf.Batch([ctx], [b[0]], [b[1]], [b[2]], [b[3]], [b[4]])
    batch.launch()
    batch.sync()
    ref = b[3].cpu().numpy().copy(), b[4].cpu().numpy().copy()
    g = np.random.default_rng(k)
    nb = 3 * w.ncol
    off = np.concatenate([[0], np.cumsum(g.integers(0, 40, nb))]).astype(np.int64)
    t = int(off[-1])
    prob = (off, g.standard_normal((t, k)), np.ones(t, np.float32), g.standard_normal(t), g.uniform(0.1, 1.0, t))
    tr0, w0 = ctx.core_batch(*prob)
    # memory of the size that a moved buffer would have left to others
    fill = [torch.full((w.ncol * k * k,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(4)]
    b[3].zero_()
    b[4].zero_()
    torch.cuda.synchronize()
    batch.launch()
    batch.sync()
    assert np.array_equal(b[3].cpu().numpy(), ref[0]) and np.array_equal(b[4].cpu().numpy(), ref[1])
    tr, wv = ctx.core_batch(*prob)
    assert np.array_equal(tr, tr0) and np.array_equal(wv, w0)
    assert all(bool(torch.isnan(f).all()) for f in fill)
    batch.close()
