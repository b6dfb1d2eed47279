"""The allocation-free ordering's status from several host threads: calls that follow one another on the GPU (a lock around
each) report their own status, finite and non-finite positions in turn, whichever thread reads it last."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_status_is_the_calls_own():
    from fdps_sph_gb300 import lib
    L = lib.load()
    n, rounds = 3000, 60
    lock, wrong = threading.Lock(), []

    def work(bad):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            pos = torch.rand((3, n), dtype=torch.float64, device="cuda")
            if bad:
                pos[1, n // 2] = float("nan")
            keys, order = torch.empty(n, dtype=torch.int64, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
            stream.synchronize()
            for _ in range(rounds):
                with lock:
                    rc = L.sph_morton_order_noalloc(*(C.c_void_p(p.data_ptr()) for p in pos), n, C.c_void_p(keys.data_ptr()),
                                                    C.c_void_p(order.data_ptr()), C.c_void_p(stream.cuda_stream))
                if rc != (-5 if bad else lib.SPH_OK):
                    wrong.append((bad, rc))

    threads = [threading.Thread(target=work, args=(k % 2 == 1,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
