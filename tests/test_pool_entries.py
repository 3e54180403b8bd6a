"""Entries of the list pool from the free memory (lg_pool_entries, host code): a device
with room takes the core's intermediates off, one that is short of memory gives them
at most half of what 1 GiB for the rest of the run leaves, and a pool that is held
counts as free."""
import ctypes as C

import pytest

from conftest import pkg

GIB = 1 << 30


@pytest.fixture(scope="module")
def entries():
    pkg("build").build()
    f = pkg("letkf").load_library().lg_pool_entries
    f.argtypes, f.restype = [C.c_int64] * 4, C.c_int64
    return f


@pytest.mark.parametrize("free,held,scratch,entry,want", [
    (270 * GIB, 0, 2 * GIB, 12, 267 * GIB // 12),
    (260 * GIB, 10 * GIB, 2 * GIB, 20, 267 * GIB // 20),
    (5 * GIB, 0, 2 * GIB, 12, 2 * GIB // 12),
    # less than the intermediates want: half of the rest, not nothing
    (3 * GIB, 0, 2 * GIB, 12, 1 * GIB // 12),
    (2 * GIB, 0, 2 * GIB, 12, GIB // 2 // 12),
    (GIB + 24, 0, 2 * GIB, 12, 1),
    (GIB, 0, 0, 12, 1),
    (0, 0, 2 * GIB, 12, 1),
    (2 * GIB, 0, 0, 12, GIB // 12),
])
def test_entries(entries, free, held, scratch, entry, want):
    assert entries(free, held, scratch, entry) == want
