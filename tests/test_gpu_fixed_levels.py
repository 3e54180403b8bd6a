"""lg_fx_levels (letkf_fixed.cuh) on level sums over the whole range that 64 products
of digits can reach: within half a unit (and FP32's rounding of the last two levels'
sum) of the integer they stand for."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

SRC = r"""
#include "letkf_fixed.cuh"
__global__ void k_levels(int n, const float *s, long long *v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x[7];
    for (int l = 0; l < 7; l++) x[l] = s[7 * i + l];
    v[i] = lg_fx_levels(x);
}
extern "C" int levels(int n, const float *s, long long *v)
{
    k_levels<<<(n + 127) / 128, 128>>>(n, s, v);
    return (int)cudaDeviceSynchronize();
}
"""
# (level 0 alone would reach 2^18, but the whole stays within 2^62: Cauchy-Schwarz over 64 operands)
MOST = [2 ** 17, 2 ** 21, 6291456, 10485760, 14680064, 18874368, 20971520]


def test_whole_range(tmp_path):
    torch = pytest.importorskip("torch")
    b = pkg("build")
    src, lib = tmp_path / "levels.cu", tmp_path / "levels.so"
    src.write_text(SRC)
    subprocess.run([b.nvcc(), *b.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-cudart", "shared",
                    "-Xlinker", f"-rpath,{os.path.join(b.CUDA_HOME, 'lib64')}", "-I", b.CSRC, str(src), "-o", str(lib)],
                   check=True, capture_output=True)
    g = np.random.default_rng(0)
    n = 20000
    most = np.array(MOST, dtype=np.float64)
    s = np.rint(g.uniform(-1, 1, (n, 7)) * most)
    s[:128] = most * np.array([[1 if i >> l & 1 else -1 for l in range(7)] for i in range(128)])
    s[128:256] = np.sign(s[:128]) * (2 ** 22 + np.arange(128)[:, None] - 64)
    s[128:256, :2] = s[:128, :2]
    s[:, 4:] = s[:, 4:].astype(np.float32)                # sums past 2^24 are FP32 values
    v = np.empty(n, dtype=np.int64)
    ds = torch.from_numpy(np.ascontiguousarray(s, dtype=np.float32)).cuda()
    dv = torch.empty(n, dtype=torch.int64, device="cuda")
    L = C.CDLL(str(lib))
    torch.cuda.synchronize()
    assert L.levels(n, C.c_void_p(ds.data_ptr()), C.c_void_p(dv.data_ptr())) == 0
    v = dv.cpu().numpy()
    for i in range(n):
        exact = sum(int(s[i, l]) << (9 * (6 - l)) for l in range(7))        # units of 2^-9
        tol = 256 + (512 if abs(s[i, 5]) > 2 ** 23 else 256)
        assert abs((int(v[i]) << 9) - exact) <= tol, (i, s[i], v[i])
