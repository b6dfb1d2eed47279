"""FP64 functor kernels against the functors' own loops in numpy, at the sizes where the blocks (32 i-particles),
the tiles (512 j) and the 32-entry queues have their edges.

Tolerance: a sum of N terms t accumulated in any order in FP64, each term evaluated with at most 64 roundings, is
within (N + 64) 2^-53 sum |t| of the exact value; the epilogues add a few roundings (1e-14 relative on top)."""
import numpy as np
import pytest

from fdps_sph_gb300 import layouts as T

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _walk(kind, ni, nj, seed, spread=1.0):
    """ni i-particles in a unit-density cluster (h about 1.2 spacings) and nj j around it: about half of them
    beyond every support"""
    rng = np.random.default_rng(seed)
    from fdps_sph_gb300 import lib
    I, J = np.zeros(ni, lib._KINDS[kind][0]), np.zeros(nj, lib._KINDS[kind][1])
    side = max(ni, 1) ** (1 / 3) * 1.0e5
    off = np.array([3.0e7, -1.0e7, 2.0e6])
    I["pos"] = off + rng.uniform(0, side, (ni, 3))
    J["pos"] = off + rng.uniform(-4.0e5 * spread, side + 4.0e5 * spread, (nj, 3))
    k = min(ni, nj)
    J["pos"][:k] = I["pos"][:k]     # the i-particles themselves
    m = 6.0e24 / 1.0e6
    J["mass"] = m * rng.uniform(0.5, 2.0, nj)
    h = 1.2e5
    if kind != "grav":
        I["smth"], J["smth"] = h * rng.uniform(0.8, 1.2, ni), h * rng.uniform(0.8, 1.2, nj)
    if kind == "dens":
        I["mass"] = m
    if kind in ("drvt", "hydro"):
        I["vel"], J["vel"] = rng.normal(0, 500.0, (ni, 3)), rng.normal(0, 500.0, (nj, 3))
        J["vel"][:k] = I["vel"][:k]
        I["dens"] = rng.uniform(3000, 9000, ni)
    if kind == "hydro":
        J["dens"] = rng.uniform(3000, 9000, nj)
        for a, n in ((I, ni), (J, nj)):
            a["pres"], a["snds"] = rng.normal(1e11, 1e10, n), rng.uniform(3e3, 9e3, n)
            a["grad_smth"], a["Bal"], a["AVa"] = rng.uniform(0.9, 1.1, n), rng.uniform(0, 1, n), 1.0
    if kind == "grav":
        I["eps2"] = (h * rng.uniform(0.8, 1.2, ni)) ** 2
    return I, J


def _wend(r, H):
    s = r / H
    p = np.maximum(1 - s, 0)
    n = (1365 / 64) / (H ** 3 * np.pi)
    return n * (1 + s * (8 + s * (25 + s * 32))) * p ** 8, n * -22 * s * (1 + s * (7 + s * 16)) * p ** 7 / (r * H + 4e-7 * H)


def _reference(kind, I, J, S):
    """sums and sums of magnitudes over the whole list, per output"""
    if kind == "grav":
        P = np.concatenate([J["pos"], S["pos"]])
        m = np.concatenate([J["mass"], S["mass"]]) * 6.67e-11
        d = I["pos"][:, None] - P
        ri = 1 / np.sqrt((d * d).sum(2) + I["eps2"][:, None])
        a = -(m * ri ** 3)[..., None] * d
        t = dict(pot=-m * ri, **{f"a{k}": a[..., k] for k in range(3)})
        return {k: (v.sum(1), np.abs(v).sum(1)) for k, v in t.items()}
    d = I["pos"][:, None] - J["pos"]
    r2 = (d * d).sum(2)
    r = np.sqrt(r2)
    w, g = _wend(r, 2.5 * I["smth"][:, None])
    m = J["mass"]
    if kind == "dens":
        t = dict(dens=m * w)
        return {k: (v.sum(1), np.abs(v).sum(1)) for k, v in t.items()}
    v = I["vel"][:, None] - J["vel"]
    vd = (v * d).sum(2)
    avd = (np.abs(v) * np.abs(d)).sum(2)
    if kind == "drvt":
        mg = -m * g
        c = np.cross(v, d)
        ac = np.stack([np.abs(v[..., (k + 1) % 3] * d[..., (k + 2) % 3]) + np.abs(v[..., (k + 2) % 3] * d[..., (k + 1) % 3])
                       for k in range(3)], 2)
        out = dict(div=((mg * vd).sum(1), (np.abs(mg) * avd).sum(1)))
        for k in range(3):
            out[f"rot{k}"] = ((mg * c[..., k]).sum(1), (np.abs(mg) * ac[..., k]).sum(1))
        gs = m / I["smth"][:, None]
        out["grad"] = ((-gs * (3 * w + g * r2)).sum(1), (gs * (3 * w + np.abs(g) * r2)).sum(1))
        return out
    with np.errstate(invalid="ignore", divide="ignore"):
        wr = np.where(vd < 0, vd / r, 0)
    vs = I["snds"][:, None] + J["snds"] - 3 * wr
    av = -0.5 * vs * wr / (0.5 * (I["dens"][:, None] + J["dens"])) * 0.5 * (I["Bal"][:, None] + J["Bal"])
    _, gj = _wend(r, 2.5 * J["smth"])
    gw = 0.5 * (g * I["grad_smth"][:, None] + gj * J["grad_smth"])
    A = lambda q: q["grad_smth"] * q["pres"] / q["dens"] ** 2  # noqa: E731
    Ai, Aj = A(I)[:, None], A(J)
    c = m * (Ai * g + Aj * gj + av * gw)
    cm = m * (np.abs(Ai * g) + np.abs(Aj * gj) + np.abs(av * gw))
    out = {f"a{k}": ((-c * d[..., k]).sum(1), (cm * np.abs(d[..., k])).sum(1)) for k in range(3)}
    e = m * (Ai + 0.5 * av) * gw
    out["e"] = ((e * vd).sum(1), (m * (np.abs(Ai) + np.abs(av)) * np.abs(gw) * avd).sum(1))
    out["vmax"] = (vs.max(1) if len(J) else np.zeros(len(I)),
                   (I["snds"][:, None] + J["snds"] + 3 * np.sqrt((v * v).sum(2))).max(1) if len(J) else np.zeros(len(I)))
    return out


def _close(got, ref, n, scale=1.0):
    want, mag = ref
    tol = (n + 64) * U * mag * np.abs(scale) + 1e-14 * np.abs(want * scale) + 1e-300
    assert np.all(np.abs(got - want * scale) <= tol), np.max(np.abs(got - want * scale) / tol)


SIZES = [(1, 1), (1, 0), (2, 31), (31, 32), (32, 33), (33, 511), (85, 512), (129, 513), (256, 1100), (7, 2049)]


@pytest.mark.parametrize("kind", ["dens", "drvt", "hydro", "grav"])
def test_fp64_functors_at_block_tile_and_queue_edges(kind):
    from fdps_sph_gb300 import lib
    walks = [_walk(kind, ni, nj, 10 * ni + nj) for ni, nj in SIZES]
    spj = []
    for k, (I, J) in enumerate(walks):
        s = np.zeros((0, 1, 600)[k % 3], T.SPJ_MONO)
        rng = np.random.default_rng(k)
        s["pos"], s["mass"] = rng.normal(0, 5e7, (len(s), 3)), 1e20
        spj.append(s)
    lib.batch_precision("fp64")
    # each walk alone (one i-particle per warp) and all in one dispatch give the same bits
    res = lib.run_walks(kind, [w[0] for w in walks], [w[1] for w in walks], spj if kind == "grav" else None)
    for k, ((I, J), r) in enumerate(zip(walks, res)):
        alone = lib.run_walks(kind, [I], [J], [spj[k]] if kind == "grav" else None)[0]
        assert r.tobytes() == alone.tobytes()
        ref = _reference(kind, I, J, spj[k])
        n = len(J) + len(spj[k])
        if kind == "dens":
            want, mag = ref["dens"]
            _close(r["dens"], (np.maximum(want, 5.0), mag), n)
            np.testing.assert_allclose(r["smth"], 1.2 * (I["mass"] / r["dens"]) ** (1 / 3), rtol=1e-14)
        elif kind == "drvt":
            rho = 1 / I["dens"]
            _close(r["div_v"], ref["div"], n, rho)
            for c in range(3):
                _close(r["rot_v"][:, c], ref[f"rot{c}"], n, rho)
            want, mag = ref["grad"]
            f = I["smth"] * rho / 3
            _close(1 / r["grad_smth"], (1 + f * want, f * mag), n)
        elif kind == "hydro":
            for c in range(3):
                _close(r["acc"][:, c], ref[f"a{c}"], n)
            _close(r["eng_dot"], ref["e"], n)
            with np.errstate(divide="ignore"):
                if n:
                    _close(0.6 * I["smth"] / r["dt"], ref["vmax"], 0)
                else:
                    assert np.all(np.isinf(r["dt"]))
        else:
            for c in range(3):
                _close(r["acc"][:, c], ref[f"a{c}"], n)
            _close(r["pot"], ref["pot"], n)


def test_fp64_hydro_signal_velocity_comes_from_any_j():
    """the fastest approach sits far outside every support, behind many slower ones"""
    from fdps_sph_gb300 import lib
    I, J = _walk("hydro", 40, 1300, 5, spread=30.0)
    J["pos"][1200] = I["pos"][0] + 4.0e6
    J["vel"][1200] = I["vel"][0] - 3.0e4
    J["pos"][77] = I["pos"][0] - 6.0e6
    J["vel"][77] = I["vel"][0] + 3.0e4 * (1 - 1e-7)     # the runner-up, 1e-7 slower
    lib.batch_precision("fp64")
    r = lib.run_walks("hydro", [I], [J])[0]
    _close(0.6 * I["smth"] / r["dt"], _reference("hydro", I, J, None)["vmax"], 0)


@pytest.mark.parametrize("kind,field,value", [("dens", "mass", np.inf), ("dens", "pos", np.nan), ("drvt", "vel", np.nan),
                                              ("drvt", "mass", np.inf), ("hydro", "pres", np.inf),
                                              ("hydro", "pos", np.inf), ("hydro", "dens", np.nan)])
def test_fp64_functors_carry_non_finite_j_out_of_support(kind, field, value):
    """a non-finite j reaches every i-particle's sums, as in the plain loop (0 x inf is NaN)"""
    from fdps_sph_gb300 import lib
    I, J = _walk(kind, 40, 700, 9, spread=30.0)
    J[field][650] = value
    with np.errstate(all="ignore"):
        ref = _reference(kind, I, J, None)
    lib.batch_precision("fp64")
    r = lib.run_walks(kind, [I], [J])[0]
    got = {"dens": ("dens", "dens"), "drvt": ("grad", "grad_smth"), "hydro": ("e", "eng_dot")}[kind]
    if kind == "dens":   # the floor takes a NaN sum as the functor's max does
        assert np.array_equal(np.isnan(r["dens"]) | (r["dens"] == 5.0), np.isnan(ref["dens"][0]))
    else:
        assert np.array_equal(np.isfinite(r[got[1]]), np.isfinite(ref[got[0]][0]))


@pytest.mark.parametrize("kind", ["dens", "drvt", "hydro", "grav"])
def test_mixed_functors_give_the_same_bits_in_every_block_shape(kind):
    """one walk alone and ten walks (blocks of 32 i-particles), 160 walks (blocks of 64), payload and index form"""
    from fdps_sph_gb300 import lib
    walks = [_walk(kind, ni, nj, 10 * ni + nj) for ni, nj in SIZES]
    spj = [np.zeros((0, 1, 33)[k % 3], T.SPJ_MONO) for k in range(len(walks))]
    for k, s in enumerate(spj):
        s["pos"], s["mass"] = np.random.default_rng(k).normal(0, 5e7, (len(s), 3)), 1e20
    I, J = [w[0] for w in walks], [w[1] for w in walks]
    g = kind == "grav"
    lib.batch_precision("mixed")
    try:
        ten = lib.run_walks(kind, I, J, spj if g else None)
        many = lib.run_walks(kind, 16 * I, 16 * J, 16 * spj if g else None)
        at = np.concatenate([[0], np.cumsum([len(j) for j in J])])
        ats = np.concatenate([[0], np.cumsum([len(s) for s in spj])])
        ids = [np.arange(at[k], at[k + 1], dtype=np.int32) for k in range(len(J))]
        sids = [np.arange(ats[k], ats[k + 1], dtype=np.int32) for k in range(len(J))]
        n = lib.dispatch_index(kind, 0, I, ids, np.concatenate(J), sids if g else None,
                               np.concatenate(spj) if g else None, send=True)
        index = lib.retrieve(kind, 0, n)
        for k in range(len(walks)):
            alone = lib.run_walks(kind, [I[k]], [J[k]], [spj[k]] if g else None)[0]
            assert alone.tobytes() == ten[k].tobytes() == index[k].tobytes()
            for r in range(16):
                assert many[r * len(walks) + k].tobytes() == alone.tobytes()
    finally:
        lib.batch_precision("fp64")
