"""Host arrays given back to the library: any number, of any size and from any
thread, are kept within the caches' bounds or freed."""

import ctypes as C
import threading

import rvsp_b200 as rv

KB, MB = 1 << 10, 1 << 20


def _libc():
    libc = C.CDLL(None)
    libc.malloc.restype, libc.malloc.argtypes = C.c_void_p, [C.c_size_t]
    return libc


def _resident():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * 4096


def test_many_sizes_from_many_threads():
    L, libc = rv.lib(), _libc()

    def work(k):
        for i in range(40):
            for size in (1, 100 * KB, 256 * KB, 300 * KB, (1 + (i + k) % 5) * MB, 65 * MB):
                L.rvsp_cuda_host_free(C.c_void_p(libc.malloc(size)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()


def test_what_is_kept_is_bounded():
    L, libc = rv.lib(), _libc()
    before = _resident()
    for size in (1 * MB, 40 * MB):
        for _ in range(30):
            p = libc.malloc(size)
            C.memset(p, 1, size)
            L.rvsp_cuda_host_free(C.c_void_p(p))
    assert _resident() - before < 200 * MB
