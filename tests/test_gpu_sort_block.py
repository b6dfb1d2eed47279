"""The one-block key sort (runs of at most 8,192 particles) at the edges of its warps (256 keys), rounds (32) and range,
and the permutation's field shares, against numpy's stable sort; the same runs beside one that takes the other sort."""
import numpy as np
import pytest

from helpers import device_context, tillotson_materials
from test_gpu_sort_sizes import _block, _keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[31, 32, 33, 255, 256, 257], [7935, 1, 7936, 2], [8191], [8192], [8193], [8192, 5, 8191],
                                   [8192, 8193, 31, 256]])
@pytest.mark.parametrize("equal", [False, True])
def test_block_sort(sizes, equal):
    ctx = device_context(tillotson_materials(), precision=1)
    blocks = [_block(n, 11 * k + n, equal) for k, n in enumerate(sizes)]
    hs, offs = [], np.concatenate([[0], np.cumsum(sizes)])
    for F in blocks:
        hs.append(ctx.add_run(F, np.arange(F.shape[1]) + 7, np.zeros(F.shape[1], np.int32)))
    ctx.run_pass(0)
    slot, keys = ctx.order()
    got = np.concatenate([ctx.download_run(h)[0].T[slot[a:a + F.shape[1]]] for h, F, a in zip(hs, blocks, offs)])
    at = 0
    for F in blocks:
        n = F.shape[1]
        k = _keys(F[:3])
        o = np.argsort(k, kind="stable")
        assert np.array_equal(slot[at:at + n], o)
        assert np.array_equal(keys[at:at + n], k[o])
        assert np.array_equal(got[at:at + n], F[:, o].T)   # every field through the same permutation
        at += n
