"""Where the integer forms of the double-float split and the key coordinates meet their limits: positions of tiny
magnitude (the split's normal range ends at 2^-70; squares of distances stay normal floats), zeros, ties of the
rounding, cell borders: keys against numpy's, and lists (which read the split positions) against brute force."""
import numpy as np
import pytest

from helpers import device_context, tillotson_materials
from test_gpu_sort_sizes import _keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -50, 2.0 ** 40])
@pytest.mark.parametrize("precision", [0, 1])
def test_split_and_keys(scale, precision):
    from fdps_sph_gb300 import ic
    f = ic.FIELD
    n = 1500
    rng = np.random.default_rng(3)
    F = np.zeros((len(ic.FIELDS), n))
    x = rng.uniform(-1.0, 1.0, (3, n)) * 2.0 ** rng.integers(-30, 1, (3, n))   # at 2^-50: on both sides of the limit
    x[:, :40] = 0.0
    x[0, :40] = 1.0 + np.arange(40) * 2.0 ** -25   # ties: 24 bits and a half
    x[1, 40:60] = -(1.0 + 2.0 ** -24)
    x[2, 60:90] = rng.integers(-8, 8, 30) / 8.0
    x *= scale
    F[:3] = x
    F[f["mass"]], F[f["dens"]], F[f["eng"]] = 1.0e3, 5.0, 1.0
    F[f["smth"]] = 0.1 * scale
    ctx = device_context(tillotson_materials(), precision=precision)
    ctx.upload(F, np.arange(n), np.zeros(n, np.int32))
    ctx.run_pass(0)
    slot, keys = ctx.order()
    k = _keys(x)
    o = np.argsort(k, kind="stable")
    assert np.array_equal(slot, o) and np.array_equal(keys, k[o])
    ctx.run_pass(1)
    S = x[:, o]
    H2 = (2.5 * F[f["smth"], 0]) * (2.5 * F[f["smth"], 0])
    for i in range(0, n, 7):
        d = S - S[:, [i]]
        r2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
        assert np.array_equal(ctx.neighbors(0, i), np.flatnonzero(r2 < H2)), i
