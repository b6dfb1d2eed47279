"""Mixed-precision functor kernels against the functors' own loops in numpy (FP64).

Tolerance of the gravity sums: a term m r^-3 dx has at most 28 relative errors of 2^-24 (coordinate differences of
double-floats, three squares, the approximate root and its powers, the products), and FP32 partial sums of 32 terms add
32 more: 60 x 2^-24 of the sum of |t|."""
import numpy as np
import pytest

from fdps_sph_gb300 import layouts as T
from test_gpu_batch64 import _reference, _walk

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
