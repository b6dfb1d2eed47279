"""Mixed-precision functor kernels against the functors' own loops in numpy (FP64), at the sizes where blocks (32
i-particles), partial sums (32 j) and tiles (128 j) have their edges.

Tolerance of the gravity sums: a term m r^-3 dx has at most 28 relative errors of 2^-24 (coordinate differences of
double-floats, three squares, the approximate root and its powers, the products), and FP32 partial sums of 32 terms add
32 more: 60 x 2^-24 of the sum of |t|.

Of the others: at most 48 errors a term (polynomials, two reciprocals, the artificial viscosity) and 32 of the sums, of the
magnitude |t| that the term's own differences could cancel from; and r / H has 16 at most (differences, squares, the
approximate root, 1 / H), so 16 x 2^-24 of what |t| changes by with r / H."""
import numpy as np
import pytest

from fdps_sph_gb300 import layouts as T
from test_gpu_batch64 import SIZES, _reference, _walk, _wend

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


@pytest.mark.parametrize("first,others", [(0.0, True), (0.0, False), (-0.0, True), (1.0e18, True)])
@pytest.mark.parametrize("nj,ns", [(0, 40), (70, 0), (70, 40)])
def test_mixed_gravity_takes_massless_first_entries(nj, ns, first, others):
    """the first entry of the list, whose mass the sums are scaled by, has no mass; or none has"""
    from fdps_sph_gb300 import lib
    I, J = _walk("grav", 37, nj, 3 + nj)
    S = np.zeros(ns, T.SPJ_MONO)
    S["pos"], S["mass"] = np.random.default_rng(ns).normal(0, 5e7, (ns, 3)), 1e20
    for a in (J, S):
        a["mass"] *= others
    (J if nj else S)["mass"][0] = first
    lib.batch_precision("mixed")
    try:
        r = lib.run_walks("grav", [I], [J], [S])[0]
    finally:
        lib.batch_precision("fp64")
    ref = _reference("grav", I, J, S)
    for k, got in (("pot", r["pot"]), *((f"a{c}", r["acc"][:, c]) for c in range(3))):
        want, mag = ref[k]
        assert np.all(np.abs(got - want) <= 60 * U * mag), (k, np.max(np.abs(got - want) / (mag + 1e-300)) / U)


def _magnitudes(kind, I, J, f):
    """per pair, the magnitudes of the terms' factors with nothing cancelled, all distances times f"""
    d = f * (I["pos"][:, None] - J["pos"])
    ad = np.abs(d)
    r2 = (d * d).sum(2)
    r = np.sqrt(r2)
    w, g = _wend(r, 2.5 * I["smth"][:, None])
    m, g = J["mass"], np.abs(g)
    if kind == "dens":
        return dict(dens=m * w)
    av = np.abs(I["vel"][:, None] - J["vel"])
    avd = (av * ad).sum(2)
    if kind == "drvt":
        out = {f"rot{k}": m * g * (av[..., (k + 1) % 3] * ad[..., (k + 2) % 3] + av[..., (k + 2) % 3] * ad[..., (k + 1) % 3])
               for k in range(3)}
        return dict(out, div=m * g * avd, grad=m / I["smth"][:, None] * (3 * w + g * r2))
    with np.errstate(invalid="ignore", divide="ignore"):
        wr = np.where(r > 0, avd / r, 0)
    vs = I["snds"][:, None] + J["snds"] + 3 * wr
    visc = 0.5 * vs * wr / (0.5 * (I["dens"][:, None] + J["dens"])) * 0.5 * (I["Bal"][:, None] + J["Bal"])
    gj = np.abs(_wend(r, 2.5 * J["smth"])[1])
    gw = 0.5 * (g * I["grad_smth"][:, None] + gj * J["grad_smth"])
    A = lambda q: np.abs(q["grad_smth"] * q["pres"] / q["dens"] ** 2)  # noqa: E731
    Ai = A(I)[:, None]
    c = m * (Ai * g + A(J) * gj + visc * gw)
    return dict({f"a{k}": c * ad[..., k] for k in range(3)}, e=m * (Ai + 0.5 * visc) * gw * avd)


def _tolerances(kind, I, J):
    M, M1 = _magnitudes(kind, I, J, 1.0), _magnitudes(kind, I, J, 1.0 + 1e-6)
    return {k: U * (80 * v.sum(1) + 16 * (np.abs(M1[k] - v) / 1e-6).sum(1)) for k, v in M.items()}


@pytest.mark.parametrize("kind", ["dens", "drvt", "hydro", "grav"])
def test_mixed_functors_at_block_sum_and_tile_edges(kind):
    from fdps_sph_gb300 import lib
    sizes = SIZES + [(63, 31), (64, 32), (65, 33), (32, 96), (33, 127), (128, 128), (127, 129)]
    walks = [_walk(kind, ni, nj, 10 * ni + nj) for ni, nj in sizes]
    spj = [np.zeros((0, 1, 33)[k % 3], T.SPJ_MONO) for k in range(len(walks))]
    for k, s in enumerate(spj):
        s["pos"], s["mass"] = np.random.default_rng(k).normal(0, 5e7, (len(s), 3)), 1e20
    I, J = [w[0] for w in walks], [w[1] for w in walks]
    gravity = kind == "grav"
    lib.batch_precision("mixed")
    try:
        res = lib.run_walks(kind, I, J, spj if gravity else None)
    finally:
        lib.batch_precision("fp64")
    for i, j, s, r in zip(I, J, spj, res):
        ref = _reference(kind, i, j, s)
        tol = {k: 60 * U * v[1] for k, v in ref.items()} if gravity else _tolerances(kind, i, j)
        rho = None if gravity or kind == "dens" else 1 / i["dens"]
        if kind == "dens":
            got = dict(dens=r["dens"])
            ref["dens"] = (np.maximum(ref["dens"][0], 5.0), None)
        elif kind == "drvt":
            f = i["smth"] * rho / 3
            got = dict({f"rot{k}": r["rot_v"][:, k] / rho for k in range(3)}, div=r["div_v"] / rho,
                       grad=(1 / r["grad_smth"] - 1) / f)
            tol["grad"] = tol["grad"] + 4e-16 / f     # the 1 beside the sum
        elif kind == "hydro":
            got = dict({f"a{k}": r["acc"][:, k] for k in range(3)}, e=r["eng_dot"])
            if len(j):
                got["vmax"], tol["vmax"] = 0.6 * i["smth"] / r["dt"], 16 * U * ref["vmax"][1]
        else:
            got = dict({f"a{k}": r["acc"][:, k] for k in range(3)}, pot=r["pot"])
        for k, v in got.items():
            err = np.abs(v - ref[k][0])
            assert np.all(err <= tol[k] + 1e-300), (kind, len(i), len(j), k, np.max(err / (tol[k] + 1e-300)))
