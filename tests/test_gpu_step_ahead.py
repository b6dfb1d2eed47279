"""Work launched before its condition is known (EoS and lists behind a density round, kick and dt behind gravity) and
run again where the condition asks for it: the bits of a step that launches it ahead against a step that sends its
results to the host, which waits; with particles that leave their skin, and with gravity walks that need larger buffers."""
import numpy as np
import pytest

from helpers import device_context, tillotson_materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [0.5, 0.0])
@pytest.mark.parametrize("grow", [1.0, 0.9, 0.6])
def test_step_ahead(theta, grow):
    from fdps_sph_gb300 import ic, lib
    f = ic.FIELD
    F, ids, mats, _ = ic.config_small_impact(n_target=7200, n_impactor=800)
    F[f["smth"]] *= grow   # supports that grow in the density passes
    out, repairs = [], []
    for ahead in (True, False):
        ctx = device_context(tillotson_materials(), precision=1, theta=theta)
        ctx.upload(F, ids, mats)
        ctx.prologue()
        buf = np.zeros((len(lib.FIELDS), F.shape[1]))
        for k in range(3):
            D, i, m = ctx.download()
            D[f["smth"]] *= grow   # and in the step's
            ctx.upload(D, i, m, dt=1.0, forces_valid=True)
            if ahead:
                ctx.step(1)
            else:
                ctx.step_download(buf, lib.FIELDS)
        out.append(ctx.download()[0])
        c = ctx.counters()
        repairs.append(c["walks_repair"] + c["walks_full"])
    assert np.array_equal(out[0], out[1])
    assert repairs[0] == repairs[1] and (grow == 1.0 or repairs[0] > 4)
