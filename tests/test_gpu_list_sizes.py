"""Neighbour lists and densities around the sizes where the warps per walk unit (4, 2, 1) and the density's threads per
particle change (15,200, 30,400 and 50,160 particles on 152 SMs): exact sets against brute force for sampled
particles, and the same run's bits alone and beside another run, which changes the shapes but not the results."""
import numpy as np
import pytest

from helpers import by_id, device_context, tillotson_materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 15199, 15200, 30399, 30400, 50159, 50160])
@pytest.mark.parametrize("precision", [0, 1])
def test_lists_at_shape_changes(n, precision):
    from fdps_sph_gb300 import ic
    f = ic.FIELD
    F, ids, mats, _ = ic.config_small_impact(seed=n, n_target=n - n // 10, n_impactor=n // 10)
    ctx = device_context(tillotson_materials(), precision=precision, self_gravity=0)
    ctx.upload(F, ids, mats)
    ctx.prologue()
    D, i, _ = ctx.download()
    slot, _ = ctx.order()
    S = D[:, slot]
    x, h = S[:3], S[f["smth"]]
    H2 = (2.5 * h) * (2.5 * h)
    for k in np.random.default_rng(n).integers(0, n, 40):
        d = x - x[:, [k]]
        r2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
        assert np.array_equal(ctx.neighbors(0, k), np.flatnonzero(r2 < H2[k]))
        assert np.array_equal(ctx.neighbors(1, k), np.flatnonzero((r2 < H2[k]) | (r2 < H2)))


def test_runs_keep_their_bits_across_shape_changes():
    from fdps_sph_gb300 import ic
    small = ic.config_small_impact(seed=5, n_target=4500, n_impactor=503)[:3]
    big = ic.config_small_impact(seed=6, n_target=63000, n_impactor=7000)[:3]
    for precision in (0, 1):
        out = []
        for runs in ([small], [small, big], [big, small]):
            ctx = device_context(tillotson_materials(), precision=precision)
            hs = [ctx.add_run(*r) for r in runs]
            ctx.step(3)
            k = next(q for q, r in enumerate(runs) if r is small)
            X, i, _ = ctx.download_run(hs[k])
            out.append(by_id(X, i))
        assert all(np.array_equal(out[0], o) for o in out[1:])
