"""Two problems of 32 members in one root matrix of the FP64 form, one of them so
strongly observed that its FP32 eigenpairs overflow: it goes to k_core_fp64, and its
partner is bitwise what it is alone, solved by the tensor-core path."""
import numpy as np
import pytest

from test_gpu_f64_digits import _context, _problems, letkf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strong", [3e8, 1e10, 1e13, 1e16, 3e17])
@pytest.mark.parametrize("order", [0, 1])
def test_partner_out_of_range(letkf, strong, order):  # noqa: F811
    counts = [150, 150, 90, 200, 300, 31, 64, 80]
    scale = np.where(np.arange(8) % 2 == order, strong, 1.0)
    off, hx, rdi, dep, rloc = _problems(32, counts, 7, scale)
    ctx = _context(letkf, 32)
    tr, w = ctx.core_batch(off, hx, rdi, dep, rloc)
    assert ctx.general_counts() == (4, 0)
    for b in range(8):
        s = slice(off[b], off[b + 1])
        t1, w1 = ctx.core_batch(np.array([0, counts[b]]), hx[s], rdi[s], dep[s], rloc[s])
        assert ctx.general_counts() == (int(scale[b] != 1.0), 0)
        assert np.array_equal(t1[0], tr[b]) and np.array_equal(w1[0], w[b]), b
