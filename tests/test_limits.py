"""The particle counts that the C ABI takes and the memory that it asks for per particle, without a
GPU: P2G's payload places (two per particle, the top bit of a place says how its layer is laid out)
have to fit in 31 bits, and the workspace holds no space that nothing reaches."""
import ctypes as C

import pytest

from peel_mpm_b200 import _lib

MOST = (1 << 30) - 32


def _sizes(n):
    lib = _lib.load()
    out, lay = C.c_size_t(0), _lib.pm_ws_layout()
    one = (C.c_int64 * 2)(n - n // 3, n // 3), (C.c_int32 * 2)(32, 32)
    return [lib.pm_workspace_size(n, 64, C.byref(out)), lib.pm_workspace_layout(n, 64, C.byref(lay)),
            lib.pm_batch_workspace_size(2, *one, C.byref(out)), lib.pm_tape_size(n, 64, 1, 0, C.byref(out))]


@pytest.mark.parametrize("n", [0, 1, MOST])
def test_counts_whose_places_fit_are_taken(n):
    assert _sizes(n) == [_lib.PM_OK] * 4


@pytest.mark.parametrize("n", [MOST + 1, 1 << 30, (1 << 31) - 1, 1 << 31])
def test_counts_whose_places_do_not_fit_are_refused(n):
    assert _sizes(n) == [_lib.PM_ERR_ARG] * 4
