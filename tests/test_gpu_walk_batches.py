"""The superset walk's batches: leaves of one particle (32 to a step), of up to 32 and above (coincident particles), spans
that end inside a batch of 32 survivors, rows at and above a batch: the exact lists made from it against brute force."""
import numpy as np
import pytest

from helpers import device_context, tillotson_materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_leaf", [1, 8, 32])
@pytest.mark.parametrize("n,same", [(31, 0), (32, 0), (33, 0), (64, 33), (65, 32), (1500, 0), (1500, 70)])
def test_walk_batches(n_leaf, n, same):
    from fdps_sph_gb300 import ic
    f = ic.FIELD
    F, ids, mats, _ = ic.config_small_impact(seed=n, n_target=4500, n_impactor=500)
    F, ids, mats = np.ascontiguousarray(F[:, :n]), ids[:n].copy(), mats[:n].copy()
    for c in "xyz":
        F[f[c], :same] = F[f[c], 0]
    for precision in (0, 1):
        ctx = device_context(tillotson_materials(), precision=precision, n_leaf=n_leaf)
        ctx.upload(F, ids, mats)
        ctx.run_pass(0)
        slot, _ = ctx.order()
        S = ctx.download()[0][:, slot]
        x, h = S[[f["x"], f["y"], f["z"]]], S[f["smth"]]
        ctx.run_pass(1)
        H2 = (2.5 * h) * (2.5 * h)
        for k in range(0, n, max(1, n // 100)):
            d = x - x[:, [k]]
            r2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
            assert np.array_equal(ctx.neighbors(0, k), np.flatnonzero(r2 < H2[k])), (precision, k)
