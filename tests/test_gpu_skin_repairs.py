"""Exact lists after repairs of the neighbour rows between FP64 passes, against brute force, where one particle j changes its h twice inside the
skin (a factor 1.06 before its rows are walked again) while a particle v that leaves its own has some units walked again.

``grows``: j, among light particles close by, grows by 1.05 in every density pass; v shares its unit.  Particle i in the
other unit is 1.09 of j's first support away: outside the rows as first walked, inside j's support after two passes.
``dips``: j shrinks to 0.9 and comes back to 1.05 of its first h (a heavy particle at 0.576 of its support, whose weight
falls quickly); v shares i's unit, whose rows are walked again while j is small.  i is one first support of j away.

Lengths are in units of j's first h.  A particle without neighbours and with the density floor (5) keeps
h = 1.2 (m / 5)^(1/3), or grows to it by at most 1.58 a pass."""
import numpy as np
import pytest

from helpers import device_context, tillotson_materials

pytestmark = pytest.mark.gpu
H0 = 1.0e5


def _cap(m):
    return 1.2 * (m / 5.0) ** (1.0 / 3.0)


def _w(s):
    return (1 + s * (8 + s * (25 + s * 32))) * (1 - s) ** 8


def _scene(case):
    """rows of x, y, z, mass, h in units of H0 and H0^3, and the numbers of j and i"""
    rng = np.random.default_rng(5)
    light = 5.0 * (0.1 / 3.0) ** 3                # support 0.1
    rows = []
    m = 8.0 if case == "grows" else 6.0           # j's cap is above what it grows to
    d = 2.5 * (1.09 if case == "grows" else 1.0)  # distance from j to i
    j, i, v = (-d / 2, -0.05, -0.05), (d / 2, -0.05, -0.05), [0, -0.05, -0.05]
    rows.append((*j, m, 1.0))
    rows.append((*i, light, _cap(light)))
    v[0] = j[0] - 0.5 if case == "grows" else i[0] + 0.5
    rows.append((*v, light, _cap(light) / 1.2))   # leaves its skin in the first pass
    if case == "grows":
        for _ in range(24):   # shrinking, since their own mass is small
            p = np.array(j) + 0.02 * rng.uniform(-1, 1, 3)
            rows.append((*p, 2.4355 * m / 24, 0.5))
    else:
        s = 0.576
        rows.append((j[0], j[1] - 2.5 * s, j[2], 4.4554 * m / _w(s), _cap(4.4554 * m / _w(s))))
    # each side of x = 0 is its own units (more than 32 particles together): 16 others, and a corner of the box
    for side in (-1, 1):
        rows.append((side * 30.0, side * 30.0, side * 30.0, light, _cap(light)))
        rows += [(side * 5.0, -1.0 - 0.5 * k, -20.0, light, _cap(light)) for k in range(16)]
    return np.array(rows).T


@pytest.mark.parametrize("case", ["grows", "dips"])
def test_lists_after_repairs(case):
    from fdps_sph_gb300 import ic, lib
    f = ic.FIELD
    R = _scene(case)
    n = R.shape[1]
    F = np.zeros((lib.NFIELD, n))
    for k, c in enumerate("xyz"):
        F[f[c]] = R[k] * H0
    F[f["mass"]], F[f["smth"]] = R[3] * H0 ** 3, R[4] * H0
    F[f["dens"]] = 5.0
    ctx = device_context(tillotson_materials(), precision=0, self_gravity=0)
    ctx.upload(F)
    ctx.run_pass(0)
    slot, _ = ctx.order()
    at = np.argsort(slot)
    h = []
    for p in range(2):
        ctx.run_pass(1)
        h.append(ctx.download()[0][f["smth"]] / H0)
    # the scene does what it says
    want = (1.05, 1.1025) if case == "grows" else (0.9, 1.05)
    assert abs(h[0][0] - want[0]) < 2e-3 and abs(h[1][0] - want[1]) < 4e-3
    assert h[0][2] > 1.06 * R[4][2] and ctx.counters()["walks_repair"] == 1
    ctx.run_pass(4)   # the symmetric lists
    S = ctx.download()[0][:, slot]
    x, H2 = S[:3], (2.5 * S[f["smth"]]) * (2.5 * S[f["smth"]])
    d = x[:, :, None] - x[:, None, :]
    r2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
    inside = (r2 < H2[:, None]) | (r2 < H2[None, :])
    assert inside[at[1], at[0]]
    for k in range(n):
        assert np.array_equal(ctx.neighbors(1, k), np.flatnonzero(inside[k])), (k, at[0], at[1])
