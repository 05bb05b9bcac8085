"""Products on a device with little memory left: what runs with C and the
operands' own structures beside it, but not with slots or segment lists too,
gives these up and returns the same C.

Each case is a process of its own (pools and plans keep memory): it takes all
but a few hundred MB of the device, calls the product, gives the memory back
and calls it again for the C to compare with."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _strata(rows, per, cols, g):
    """CSR of `per` columns a row, one in each of `per` strata of the columns."""
    import torch as T

    w = cols // per
    c = T.randint(0, w, (rows, per), generator=g, device="cuda", dtype=T.int32)
    c += T.arange(per, device="cuda", dtype=T.int32) * w
    rp = T.arange(rows + 1, device="cuda", dtype=T.int32) * per
    v = T.rand(rows * per, generator=g, device="cuda") * 2 - 1
    return rows, cols, rp, c.reshape(-1), v


def _call(fn, algo, A, B, vdtype):
    import ctypes as C

    import rvsp_b200 as rv
    import torch as T

    prp, pci, pv, nnz = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_int32()
    ops = [rv.ptr(x) for x in A[2:] + B[2:]]
    outs = [C.byref(x) for x in (prp, pci, pv, nnz)]
    if fn == "f32":
        st = rv.lib().rvsp_cuda_spgemm_f32(algo, A[0], A[1], B[1], *ops, *outs, None)
    else:
        st = rv.lib().rvsp_cuda_spgemm_f64(A[0], A[1], B[1], *ops, *outs)
    rv.check(st, fn)

    class View:
        def __init__(self, p, n, kind):
            self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (p, False),
                                             "version": 3}

    return tuple(T.as_tensor(View(p.value, n, k), device="cuda") for p, n, k in
                 ((prp, A[0] + 1, "<i4"), (pci, nnz.value, "<i4"),
                  (pv, nnz.value, "<f8" if vdtype == T.float64 else "<f4")))


def _release(c):
    import rvsp_b200 as rv

    for x in c:
        rv.free_device(x.data_ptr())


def _child(case, mb):
    import rvsp_b200 as rv
    import torch as T

    g = T.Generator(device="cuda")
    g.manual_seed(3)
    fn, algo = "f32", rv.RVSP_CUDA_ALGO_EXACT
    if case == "oneshot":  # 410 MB of slots, 410 of C
        A, B = _strata(200000, 16, 65536, g), _strata(65536, 16, 65536, g)
    if case == "f64":  # 1230 MB of slots, 440 of C
        fn = "f64"
        A, B = _strata(200000, 32, 65536, g), _strata(65536, 16, 192, g)
    small = _strata(512, 4, 512, g)
    if fn == "f64":
        A, B, small = ((*M[:4], M[4].double()) for M in (A, B, small))
    vd = A[4].dtype
    _release(_call(fn, algo, small, small, vd))  # the library and its kernels are loaded
    T.cuda.synchronize()
    hog = T.empty(T.cuda.mem_get_info()[0] - mb * MB, dtype=T.uint8, device="cuda")
    got = _call(fn, algo, A, B, vd)
    del hog
    T.cuda.empty_cache()
    want = _call(fn, algo, A, B, vd)
    for x, y in zip(got, want):
        assert T.equal(x, y)
    assert int(got[0][-1]) == got[1].numel() > 1000000
    print("same", got[1].numel())


@pytest.mark.parametrize("case,mb", [("oneshot", 640), ("f64", 1200), ("f64", 1450)])
def test_little_memory(gpu_lib, case, mb):
    import torch as T

    T.cuda.empty_cache()
    here = os.path.dirname(os.path.abspath(__file__))
    path = os.pathsep.join([here, os.path.join(os.path.dirname(here), "rv-sparse_b200"),
                            os.environ.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, os.path.abspath(__file__), case, str(mb)], text=True,
                       capture_output=True, timeout=300, env={**os.environ, "PYTHONPATH": path})
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("same")


if __name__ == "__main__":
    _child(sys.argv[1], int(sys.argv[2]))
