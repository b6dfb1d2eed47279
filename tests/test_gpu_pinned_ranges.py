"""Host blocks pinned as a whole, in adjoining pieces, and with ordinary pages between two registrations (which the copy
engine refuses and a GPU that reads pageable memory takes): the bytes of uploads and downloads."""
import ctypes as C
import mmap

import numpy as np
import pytest

from helpers import device_context, tillotson_materials

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
PAGE = 65536          # bytes; a multiple of every page size
N = 4 * PAGE // 8     # particles: a row is four such pages


class Arena:
    """zeroed pages for NFIELD rows, some of them registered"""

    def __init__(self, rows, pieces):
        self.map = mmap.mmap(-1, rows * N * 8 + PAGE)
        at = C.addressof(C.c_char.from_buffer(self.map))
        skip = -at % PAGE
        self.base = at + skip
        self.F = np.frombuffer(self.map, np.float64, rows * N, skip).reshape(rows, N)
        self.regs = []
        rt = torch.cuda.cudart()
        for a, b in pieces:   # in pages
            assert int(rt.cudaHostRegister(self.base + a * PAGE, (b - a) * PAGE, 0)) == 0
            self.regs.append(self.base + a * PAGE)

    def close(self):
        for a in self.regs:
            assert int(torch.cuda.cudart().cudaHostUnregister(a)) == 0


@pytest.mark.parametrize("pinned", ["not", "whole", "gap", "pieces"])
def test_blocks_pinned_in_pieces(pinned):
    from fdps_sph_gb300 import lib
    torch.zeros(1, device="cuda")
    rows = lib.NFIELD
    pages = rows * 4
    pieces = {"not": [], "whole": [(0, pages)], "gap": [(0, 8), (12, pages)], "pieces": [(0, 8), (8, 12), (12, pages)]}[pinned]
    rng = np.random.default_rng(1)
    F = rng.normal(1.0, 0.3, (rows, N))
    F[lib.FIELD["mass"]] = 1.0e18
    F[lib.FIELD["smth"]] = 0.01
    L = lib.load()
    src, dst = Arena(rows, pieces), Arena(rows, pieces)
    try:
        src.F[:] = F
        ctx = device_context(tillotson_materials(), precision=0, self_gravity=0)
        ctx._check(L.sph_upload(ctx.h, N, C.c_void_p(src.base), N, None, None, 0.0, 1.0, 2))
        ctx.n = N
        assert np.array_equal(ctx.download()[0], F)
        ctx.run_pass(0)
        want = ctx.download()[0]
        before = ctx.counters()["launches"]
        ctx._check(L.sph_download(ctx.h, C.c_void_p(dst.base), N, None, None))
        assert np.array_equal(dst.F, want)
        if pinned != "gap":   # inverse order and gather, or the unpermutation for the copy engine
            assert ctx.counters()["launches"] - before == (1 if pinned == "not" else 2)
    finally:
        src.close()
        dst.close()
