"""Mixed derivative and hydro sums at every kind of row length (eight entries a round, flushed every 32): n particles
within one support, so each row holds all of them, the sums in one thread's order against those of the tuned shapes
(2 and 4 threads per particle, other orders of the same FP32 terms).

Tolerance: both sides add the same terms t, FP32 partial sums of at most 32 terms per thread and then compensated, so
each is within 32 x 2^-24 sum |t| of their sum: 64 x 2^-24 sum |t| between them, sum |t| evaluated here in FP64."""
import numpy as np
import pytest

from helpers import by_id, device_context, tillotson_materials

pytestmark = pytest.mark.gpu


def _magnitudes(S, f):
    """per particle: sums of the magnitudes of the terms of div v, rot v, du/dt and the acceleration"""
    X = lambda k: S[f[k]]  # noqa: E731
    pos, vel = (np.stack([X(p + c) for c in "xyz"], 1) for p in ("", "v"))
    d, v = pos[:, None] - pos, vel[:, None] - vel
    r = np.sqrt((d * d).sum(2))

    def grad(H):
        s = r / H
        n = (1365 / 64) / (H ** 3 * np.pi)
        return np.abs(n * -22 * s * (1 + s * (7 + s * 16)) * np.maximum(1 - s, 0) ** 7 / (r * H + 4e-7 * H))

    gi, gj = grad(2.5 * X("smth")[:, None]), grad(2.5 * X("smth"))
    vd = (v * d).sum(2)
    m, rho, c, fh = X("mass"), X("dens"), X("snds"), X("grad_smth")
    curl = np.abs(np.cross(v, d))
    mg = m * gi / rho[:, None]
    with np.errstate(invalid="ignore", divide="ignore"):
        w = np.where(vd < 0, vd / r, 0)
    av = np.abs(0.5 * (c[:, None] + c - 3 * w) * w / (0.5 * (rho[:, None] + rho)) * 0.5 * (X("bal")[:, None] + X("bal")))
    gw = 0.5 * (gi * np.abs(fh)[:, None] + gj * np.abs(fh))
    A = np.abs(fh * X("pres") / rho ** 2)
    cm = m * (A[:, None] * gi + A * gj + av * gw)
    out = {"div_v": (mg * np.abs(vd)).sum(1), "eng_dot": (m * (A[:, None] + 0.5 * av) * gw * np.abs(vd)).sum(1)}
    for k, x in enumerate("xyz"):
        out["rot_" + x] = (mg * curl[..., k]).sum(1)
        out["a" + x] = (cm * np.abs(d[..., k])).sum(1)
    return out


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 15, 31, 32, 33, 40, 63, 64, 65, 96, 97, 129, 300])
def test_mixed_rows_of_every_length(n):
    from fdps_sph_gb300 import ic
    f = ic.FIELD
    rng = np.random.default_rng(n)
    F = np.zeros((len(ic.FIELDS), n))
    h = 2.4e5
    F[:3] = rng.uniform(-0.5 * h, 0.5 * h, (3, n)) + np.array([[2.0e7], [-1.0e7], [3.0e6]])   # box diagonal < 2.5 h
    F[3:6] = rng.normal(0, 300.0, (3, n))
    F[f["mass"]] = 5000.0 * h ** 3 / n
    F[f["smth"]], F[f["eng"]], F[f["ava"]], F[f["bal"]], F[f["grad_smth"]] = h, 1.0e6, 1.0, 1.0, 1.0
    ids, mats = np.arange(n), (np.arange(n) % 2).astype(np.int32)
    ctx = device_context(tillotson_materials(), precision=1, n_dens_iter=1)
    ctx.upload(F, ids, mats)
    ctx.prologue()
    assert max(len(ctx.neighbors(1, k)) for k in range(n)) == n
    S, i, _ = ctx.download()
    S = by_id(S, i)
    mag = _magnitudes(S, f)
    for tpi in (2, 4):
        ctx.set_tune(tpi, 1)
        ctx.run_pass(3)
        D, i, _ = ctx.download()
        D = by_id(D, i)
        ctx.set_tune(1, 1)
        ctx.run_pass(3)   # the hydro comparison reads one thread's derivative
        ctx.set_tune(1, tpi)
        ctx.run_pass(4)
        H, i, _ = ctx.download()
        H = by_id(H, i)
        for T, names in ((D, ("div_v", "rot_x", "rot_y", "rot_z")), (H, ("ax", "ay", "az", "eng_dot"))):
            for k in names:
                tol = 64 * 2.0 ** -24 * mag[k]
                assert np.all(np.abs(T[f[k]] - S[f[k]]) <= tol), (tpi, k)
        assert np.array_equal(H[f["dt"]], S[f["dt"]])   # a maximum, the same in any order
