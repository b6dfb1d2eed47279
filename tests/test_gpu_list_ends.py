"""Exact lists where (2.5 h)^2 overflows an FP32 number: every particle is a neighbour of every other, and the lanes of a
warp past a row's end (rows of 40 and 700 entries: 24 and 4 lanes in the last 32) add nothing, neither to the row nor, from a
spill range (rows above 512 entries), to the next one."""
import numpy as np
import pytest

from helpers import device_context, tillotson_materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [40, 700])
def test_rows_end_at_their_length_when_h_squared_overflows(n, precision):
    from fdps_sph_gb300 import ic
    f = ic.FIELD
    F, ids, mats, _ = ic.config_small_impact(seed=n, n_target=900, n_impactor=100)
    F, ids, mats = np.ascontiguousarray(F[:, :n]), ids[:n].copy(), mats[:n].copy()
    F[f["smth"]] = 1.0e19     # (2.5e19)^2 is above the largest FP32 number
    F[f["dens"]] = 3000.0
    ctx = device_context(tillotson_materials(), precision=precision, self_gravity=0)
    ctx.upload(F, ids, mats)
    ctx.run_pass(0)
    for mode, run in ((0, 3), (1, 4)):   # the derivative's gather lists, the hydro pass's symmetric ones
        ctx.run_pass(run)
        for k in range(n):
            assert np.array_equal(ctx.neighbors(mode, k), np.arange(n)), (mode, k)
