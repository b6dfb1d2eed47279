"""FP64 passes at the edges of their blocks (32 i-particles of 8 threads; gravity: up to 32 i-particles, tiles of 512
list entries), against the oracle.  Tolerances: the passes' parity bounds (1e-12 density, 1e-10 forces), floored at
the RMS."""
import numpy as np
import pytest

from helpers import by_id, device_context, oracle_config, scalar_err_rms, tillotson_materials, vec_err_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 31, 32, 33, 255, 257, 513, 1100, 3001])
def test_fp64_forces_at_block_edges(n):
    from fdps_sph_gb300 import ic
    from oracle import pyoracle as po
    rng = np.random.default_rng(n)
    f = po.FIELD
    F = np.zeros((len(ic.FIELDS), n))
    side = n ** (1 / 3) * 2.0e5
    F[:3] = rng.uniform(-side, side, (3, n)) + np.array([[2.0e7], [-1.0e7], [3.0e6]])
    F[3:6] = rng.normal(0, 300.0, (3, n))
    F[f["mass"]] = 5000.0 * 8.0e15
    F[f["smth"]] = 2.4e5
    F[f["eng"]], F[f["ava"]], F[f["bal"]], F[f["grad_smth"]] = 1.0e6, 1.0, 1.0, 1.0
    ids, mats = np.arange(n), (np.arange(n) % 2).astype(np.int32)
    ml = tillotson_materials()
    ctx = device_context(ml, precision=0)
    ctx.upload(F, ids, mats)
    ctx.prologue()
    Fd, idd, _ = ctx.download()
    Fd = by_id(Fd, idd)
    s = po.OracleSystem(F, ids, mats)
    s.prologue(oracle_config(ml))
    Fo, _, _ = s.by_id()
    for k in ("dens", "smth"):
        assert scalar_err_rms(Fd[f[k]], Fo[f[k]]) < 1e-12, k
    for k in ("div_v", "grad_smth", "bal", "eng_dot", "dt", "pot"):
        assert scalar_err_rms(Fd[f[k]], Fo[f[k]]) < 1e-10, k
    for a in "ag":
        v = [np.stack([X[f[a + c]] for c in "xyz"], 1) for X in (Fd, Fo)]
        assert vec_err_rms(*v) < 1e-10, a
