"""Uploads and downloads of pinned host blocks (copied by kernels) against pageable ones (copied by the copy engine):
the same bytes for every field, odd sizes, padded rows, rows at odd 8-byte offsets, field masks and single runs."""
import ctypes as C

import numpy as np
import pytest

from helpers import device_context, small_impact, tillotson_materials

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _pinned(rows, ld, shift=0):
    buf = torch.full((rows * ld + shift,), np.nan, dtype=torch.float64).pin_memory().numpy()
    return buf, buf[shift:].reshape(rows, ld)


@pytest.mark.parametrize("n,pad,shift", [(1, 0, 0), (7, 0, 1), (1000, 0, 0), (2047, 1, 0), (2049, 2, 1), (50001, 3, 1)])
@pytest.mark.parametrize("inputs_only", [False, True])
def test_pinned_blocks_carry_the_same_bytes(n, pad, shift, inputs_only):
    from fdps_sph_gb300 import lib
    rng = np.random.default_rng(n)
    F = rng.normal(1.0, 0.3, (lib.NFIELD, n))
    F[lib.FIELD["mass"]] = 1.0e18
    F[lib.FIELD["smth"]] = 0.05
    ld = n + pad
    keep, P = _pinned(lib.NFIELD, ld, shift)
    P[:, :n] = F
    L = lib.load()
    flags = 2 | (4 if inputs_only else 0)
    out = []
    for block, width in ((np.ascontiguousarray(F), n), (P, ld)):
        ctx = device_context(tillotson_materials(), precision=0, self_gravity=0)
        ctx._check(L.sph_upload(ctx.h, n, block.ctypes.data_as(C.c_void_p), width, None, None, 0.0, 1.0, flags))
        ctx.n = n
        res = [ctx.download()[0]]      # before any sort: the copy engine
        ctx.run_pass(0)                # the particles in key order
        res.append(ctx.download()[0])
        keep2, Q = _pinned(lib.NFIELD, ld, 1 - shift)
        ctx._check(L.sph_download(ctx.h, Q.ctypes.data_as(C.c_void_p), ld, None, None))
        assert np.array_equal(Q[:, :n], res[1]) and np.all(np.isnan(Q[:, n:]))
        keep3, M = _pinned(lib.NFIELD, ld, shift)
        names = ["x", "smth", "dens", "pot", "temp"]
        mask = sum(1 << lib.FIELD[k] for k in names)
        ctx._check(L.sph_download_fields(ctx.h, M.ctypes.data_as(C.c_void_p), ld, mask, None, None))
        rows = [lib.FIELD[k] for k in names]
        assert np.array_equal(M[rows, :n], res[1][rows])
        assert np.all(np.isnan(np.delete(M, rows, 0)))
        out.append(res)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    want = F.copy()
    if inputs_only:
        want[[k for k, f in enumerate(lib.FIELDS) if f not in lib.STEP_INPUT_FIELDS]] = 0.0
    assert np.array_equal(out[0][0], want)


def test_pinned_download_of_single_runs():
    from fdps_sph_gb300 import lib
    L = lib.load()
    ctx = device_context(tillotson_materials(), precision=1)
    hs = [ctx.add_run(*small_impact(n, 40, seed=n)[:3]) for n in (500, 901, 2000)]
    ctx.step(2)
    hs.append(ctx.add_run(*small_impact(7000, 40, seed=9)[:3]))   # not sorted yet
    for h in hs:
        X, ids, _ = ctx.download_run(h)
        keep, Q = _pinned(lib.NFIELD, X.shape[1])
        i2 = np.empty(X.shape[1], np.int64)
        ctx._check(L.sph_download_run(ctx.h, h, Q.ctypes.data_as(C.c_void_p), X.shape[1],
                                      i2.ctypes.data_as(C.c_void_p), None))
        assert np.array_equal(Q, X) and np.array_equal(i2, ids)
