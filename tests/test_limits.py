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


@pytest.mark.parametrize("n", [1, 1000, 1 << 20])
def test_workspace_holds_the_payload_and_no_more(n):
    """72 bytes a place (68 of payload, 4 of the particle's id), two places per particle in blocks of 32; the sort
    buffers, 20 bytes per particle and the histograms, are pm_bin's: a batch, which cannot call it, has none."""
    up = lambda v, a: (v + a - 1) // a * a
    L = _lib.workspace_layout(n, 64)
    assert L.inv_perm - L.payload == up(72 * up(2 * n, 32), 256)
    cells = 64 ** 3
    units = min(n, cells // 128)
    # after the payload: inverse permutation, unit list, places; then per cell count and split, per unit counts and list
    assert L.total - L.inv_perm == 3 * up(4 * n, 256) + up(8 * cells, 256) + up(cells, 256) + up(4 * cells // 128, 256) + \
        up(4 * units, 256)
    B = _lib.batch_workspace_layout([n], [64]).ws
    assert B.block_mask - B.keys_a <= 8 * 1024 and B.work - B.inv_perm == 256
    assert B.inv_perm - B.payload == L.inv_perm - L.payload
