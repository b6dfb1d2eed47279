"""The key sort against numpy's stable sort at the edges of its tiles (2,048 keys), its direct / scanned offsets (64
tiles per run) and with equal keys: one run, several runs and the allocation-free entry point."""
import numpy as np
import pytest

from helpers import by_id, device_context, tillotson_materials  # noqa: F401

pytestmark = pytest.mark.gpu


def _block(n, seed, equal=False):
    from fdps_sph_gb300 import ic
    rng = np.random.default_rng(seed)
    f = ic.FIELD
    F = np.zeros((len(ic.FIELDS), n))
    F[:3] = rng.normal(0, 1.0e6, (3, n)) + 1.0e7
    if equal:   # a few places only: long runs of equal keys, kept in input order
        F[:3] = F[:3, rng.integers(0, min(7, n), n)]
    F[f["mass"]], F[f["smth"]], F[f["dens"]], F[f["eng"]] = 1.0e18, 1.0e4, 5000.0, 1.0e6
    return F


def _keys(P):
    lo, hi = P.min(1), P.max(1)
    L = (hi - lo).max()
    half = (L if L > 0 else 1.0) * 0.50048828125
    base = (lo + hi) * 0.5 - half
    q = np.clip(np.floor((P - base[:, None]) * (2097152.0 / (half + half))), 0, 2097151).astype(np.uint64)
    k = np.zeros(P.shape[1], np.uint64)
    for b in range(21):
        for d in range(3):
            k |= ((q[d] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - d)
    return k


@pytest.mark.parametrize("sizes", [[1], [2], [2047], [2048], [2049], [131072], [131073], [300001], [1, 2048, 5, 4097],
                                   [140000, 17, 2048, 2049]])
@pytest.mark.parametrize("equal", [False, True])
def test_key_order(sizes, equal):
    ctx = device_context(tillotson_materials(), precision=1)
    blocks = [_block(n, 7 * k + n, equal) for k, n in enumerate(sizes)]
    for F in blocks:
        ctx.add_run(F, np.arange(F.shape[1]), np.zeros(F.shape[1], np.int32))
    ctx.run_pass(0)
    slot, keys = ctx.order()
    at = 0
    for F in blocks:
        n = F.shape[1]
        k = _keys(F[:3])
        o = np.argsort(k, kind="stable")
        assert np.array_equal(slot[at:at + n], o)
        assert np.array_equal(keys[at:at + n], k[o])
        at += n


@pytest.mark.parametrize("n", [1, 31, 2048, 2049, 60000, 131072])
@pytest.mark.parametrize("equal", [False, True])
def test_key_order_without_allocation(n, equal):
    torch = pytest.importorskip("torch")
    from fdps_sph_gb300 import lib
    F = _block(n, n, equal)
    P = torch.from_numpy(np.ascontiguousarray(F[:3])).cuda()
    keys = torch.empty(n, dtype=torch.int64, device="cuda")
    order = torch.empty(n, dtype=torch.int32, device="cuda")
    assert lib.load().sph_morton_order_noalloc(*(p.data_ptr() for p in P), n, keys.data_ptr(), order.data_ptr(), None) == 0
    k = _keys(F[:3])
    o = np.argsort(k, kind="stable")
    assert np.array_equal(order.cpu().numpy(), o)
    assert np.array_equal(keys.cpu().numpy().astype(np.uint64), k[o])
