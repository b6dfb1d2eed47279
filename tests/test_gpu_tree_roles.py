"""The octree's moments, walk units and gravity groups at the sizes where their kernels split the cells (blocks of a
scan, eight climbers of a warp) and for leaves of the deepest level: monopoles bit for bit against the sums in their
stated order, groups against their rule, neighbour lists (which need every particle in one unit) against brute force."""
import numpy as np
import pytest

from helpers import device_context, tillotson_materials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,same", [(1, 0), (2, 0), (8, 0), (9, 0), (33, 0), (255, 0), (257, 0), (4097, 0), (40, 40),
                                    (700, 300), (3000, 290)])
def test_tree_roles(n, same):
    from fdps_sph_gb300 import ic
    f = ic.FIELD
    F, ids, mats, _ = ic.config_small_impact(seed=n, n_target=4500, n_impactor=500)
    F, ids, mats = np.ascontiguousarray(F[:, :n]), ids[:n].copy(), mats[:n].copy()
    for c in "xyz":
        F[f[c], :same] = F[f[c], 0]   # coincident particles: a leaf of the deepest level
    ctx = device_context(tillotson_materials(), precision=0, n_group=256)
    ctx.upload(F, ids, mats)
    ctx.run_pass(0)
    slot, _ = ctx.order()
    S = ctx.download()[0][:, slot]
    t = ctx.tree()
    start, count, nch = t["start"], t["count"], t["n_child"]
    nc = len(start)
    first = np.full(nc, -1)
    parent = np.full(nc, -1)
    nxt = 1
    for c in range(nc):   # cells are stored level by level, children of one cell together
        if nch[c]:
            first[c] = nxt
            parent[nxt:nxt + nch[c]] = c
            nxt += nch[c]
    assert nxt == nc
    mom = np.zeros((nc, 4))
    for c in range(nc - 1, -1, -1):
        v = np.zeros(4)
        if nch[c]:
            for k in range(first[c], first[c] + nch[c]):
                v = v + mom[k]
        else:
            for j in range(start[c], start[c] + count[c]):
                m = S[f["mass"], j]
                v = v + np.array([m * S[f["x"], j], m * S[f["y"], j], m * S[f["z"], j], m])
        mom[c] = v
    assert np.array_equal(t["com"][:, 3], mom[:, 3])
    assert np.array_equal(t["com"][:, :3], mom[:, :3] / mom[:, 3:])
    up = np.where(parent < 0, 1 << 30, count[np.maximum(parent, 0)])
    group = np.flatnonzero(np.where(count <= 256, up > 256, nch == 0))
    ctx.run_pass(5)
    assert ctx.n_groups() == len(group)
    for g, c in enumerate(group):
        q = ctx.grav_list(g)
        assert (q["start"], q["count"]) == (start[c], count[c])
    ctx.run_pass(1)
    x, h = S[[f["x"], f["y"], f["z"]]], S[f["smth"]]
    H2 = (2.5 * h) * (2.5 * h)
    for k in range(0, n, max(1, n // 60)):
        d = x - x[:, [k]]
        assert np.array_equal(ctx.neighbors(0, k), np.flatnonzero((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2] < H2[k]))
