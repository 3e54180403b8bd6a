"""Device arrays of the FP64 form that start on an 8-byte boundary between 16-byte
ones (a view into a larger tensor): plain, overlapped and vertical-block runs take
them, with the analysis of the aligned run to the FP64 form's 1e-10."""
import numpy as np
import pytest

from conftest import field_rel_err, pkg

pytestmark = pytest.mark.gpu


def _at(torch, a, odd):
    """A device copy of a that starts `odd` doubles after a 16-byte boundary."""
    t = torch.zeros(a.size + 2, dtype=torch.float64, device="cuda")
    v = t[odd:odd + a.size].view(a.shape)
    v.copy_(torch.from_numpy(a))
    assert v.data_ptr() % 16 == 8 * odd
    return v


@pytest.mark.parametrize("k,kw", [(32, {}), (64, {}), (96, {}), (32, dict(cube_n=3, overlap=1)),
                                  (48, dict(h_mode=0, vert_dist=0.5, cube_nz=2))])
@pytest.mark.parametrize("odd_in,odd_out", [(1, 0), (0, 1), (1, 1)])
def test_arrays_between_16_byte_boundaries(k, kw, odd_in, odd_out):
    torch = pytest.importorskip("torch")
    pkg("build").build()
    letkf = pkg("letkf")
    letkf.load_library()
    w = pkg("synthetic").small_case(nlat=8, nlon=16, nz=3, k=k, nobs=300, loc_dist_km=1200.0, seed=k,
                                    h_mode=kw.get("h_mode", 1))
    ctx = letkf.LetkfGPU.from_workload(w, **kw)
    obs = letkf.ObsArrays({key: torch.from_numpy(np.ascontiguousarray(v)).cuda() for key, v in w.obs.items()},
                          device=True)
    out = []
    for i, o in ((0, 0), (odd_in, odd_out)):
        xb, axb = _at(torch, w.xb, i), _at(torch, w.axb, i)
        xa, axa = _at(torch, np.zeros_like(w.xb), o), _at(torch, np.zeros_like(w.axb), o)
        torch.cuda.synchronize()
        ctx.run_device(xb, axb, obs, xa, axa)
        torch.cuda.synchronize()
        out.append((xa.cpu().numpy(), axa.cpu().numpy()))
    assert max(field_rel_err(out[1][0], out[0][0], w).values()) <= 1e-10
    assert max(field_rel_err(out[1][1], out[0][1], w).values()) <= 1e-10
