"""Where the members entry point splits the state beside the caller's arrays (lg_split_fits,
host code): only if the observations and 2 GiB for the rest of the run fit beside it."""
import ctypes as C

import pytest

from conftest import pkg

GIB = 1 << 30


@pytest.fixture(scope="module")
def fits():
    pkg("build").build()
    f = pkg("letkf").load_library().lg_split_fits
    f.argtypes, f.restype = [C.c_int64] * 4, C.c_int
    return f


@pytest.mark.parametrize("room,split,nobs,k,want", [
    (270 * GIB, 7 * GIB, 200_000, 64, 1),
    # two states of the caller's and two of the split's fill the device: observations
    # and lists would not fit any more
    (141 * GIB, 140 * GIB, 200_000, 64, 0),
    (143 * GIB, 140 * GIB, 200_000, 64, 1),
    (143 * GIB, 140 * GIB, 5_000_000, 64, 0),
    (2 * GIB + 1000, 1000, 0, 32, 1),
    (2 * GIB + 999, 1000, 0, 32, 0),
    (0, 1000, 0, 32, 0),
])
def test_fits(fits, room, split, nobs, k, want):
    assert fits(room, split, nobs, k) == want
