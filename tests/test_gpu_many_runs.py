"""More runs in a context than a grid's second extent holds (65,535), one of them long enough for the sort of many tiles
(above 64 tiles of 2,048): every run in key order."""
import ctypes as C

import numpy as np
import pytest

from helpers import device_context, tillotson_materials

pytestmark = pytest.mark.gpu
ONES, LONG = 65_536, 64 * 2048 + 1


def test_more_runs_than_a_grid_is_high():
    from fdps_sph_gb300 import lib
    rng = np.random.default_rng(3)
    ctx = device_context(tillotson_materials(), precision=0, self_gravity=0)
    L, h = lib.load(), C.c_int64()
    blocks = []
    for n in (LONG, 1):
        F = np.zeros((lib.NFIELD, n))
        F[:3] = rng.uniform(-1e6, 1e6, (3, n))
        F[lib.FIELD["mass"]], F[lib.FIELD["smth"]], F[lib.FIELD["dens"]] = 1.0e18, 1.0e3, 3000.0
        blocks.append(F)
    x = blocks[0][:3]
    for F in [blocks[0]] + [blocks[1]] * ONES:
        ctx._check(L.sph_add_run(ctx.h, F.shape[1], F.ctypes.data_as(C.c_void_p), F.shape[1], None, None, 0.0, 0.0, 0,
                                 C.byref(h)))
    ctx.n = LONG + ONES
    ctx.run_pass(0)
    slot, keys = ctx.order()
    assert np.array_equal(np.sort(slot[:LONG]), np.arange(LONG)) and not np.any(slot[LONG:])
    assert np.all(keys[1:LONG] >= keys[:LONG - 1])
    lo, hi = x.min(1), x.max(1)
    half = (hi - lo).max() * 0.50048828125
    q = np.floor((x - ((lo + hi) * 0.5 - half)[:, None]) * (2097152.0 / (half + half))).astype(np.int64)
    top = (q[0] >> 20) << 2 | (q[1] >> 20) << 1 | q[2] >> 20     # the key's first octal digit
    assert np.array_equal(top[slot[:LONG]], (keys[:LONG] >> np.uint64(60)).astype(np.int64))
