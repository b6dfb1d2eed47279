"""The mixed path's fused gravity of small runs, whose blocks take one of a thread's two i-particles each: the same bits as
beside a run that is large enough for blocks that take both, at group sizes around a block's and a chunk's edges."""
import numpy as np
import pytest

from helpers import by_id, device_context, tillotson_materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_group", [256, 700])
def test_gravity_of_small_runs(n_group):
    from fdps_sph_gb300 import ic
    f = ic.FIELD
    big = ic.config_small_impact(seed=6, n_target=140000 * n_group // 256, n_impactor=14000)[:3]
    sizes = [1, 2, 63, 64, 65, 127, 129, 255, 257, 300, 511, 513, 700]
    small = []
    for n in sizes:
        F, ids, mats, _ = ic.config_small_impact(seed=n, n_target=1000, n_impactor=100)
        small.append((np.ascontiguousarray(F[:, :n]), ids[:n].copy(), mats[:n].copy()))

    def gravity(runs):
        ctx = device_context(tillotson_materials(), precision=1, n_group=n_group)
        hs = [ctx.add_run(*r) for r in runs]
        ctx.prologue()
        out = []
        for h in hs:
            X, i, _ = ctx.download_run(h)
            out.append(by_id(X, i)[[f["gx"], f["gy"], f["gz"], f["pot"]]])
        return out

    beside = gravity(small + [big])
    for n, r, b in zip(sizes, small, beside):
        assert np.array_equal(gravity([r])[0], b), n
