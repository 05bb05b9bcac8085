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
    if fn == "descriptor":
        a, b = (rv.csr_struct(M[0], M[1], M[3].numel(), *M[2:]) for M in (A, B))
        d = rv.Descriptor(rv.RVSP_SPGEMM_ALGO_CUDA)
        st, _, n = d.work_estimation(a, b)
        rv.check(st, "work_estimation")
        out = tuple(T.empty(k, dtype=t, device="cuda") for k, t in
                    ((A[0] + 1, T.int32), (n, T.int32), (n, T.float32)))
        c = rv.csr_struct(A[0], B[1], n, *out)
        ws = T.empty(256, dtype=T.uint8, device="cuda")
        for _ in range(2):  # the fill and a replay
            rv.check(d.compute(a, b, c, ws), fn)
        d.close()
        return out
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


def _release(fn, c):
    import rvsp_b200 as rv

    if fn != "descriptor":
        for x in c:
            rv.free_device(x.data_ptr())


def _trimmed_free():
    """Free device memory, nothing kept in the pool."""
    import ctypes as C

    import torch as T

    T.cuda.synchronize()
    cu, pool = C.CDLL("libcuda.so.1"), C.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolTrimTo(pool, C.c_size_t(0)) == 0
    return T.cuda.mem_get_info()[0]


def _kept(g):
    """What a one-shot product with 9 GB of segment lists leaves allocated, and
    that another allocation gets the memory which the pool keeps."""
    import rvsp_b200 as rv
    import torch as T

    A, B = _strata(4000, 2000, 65536, g), _strata(65536, 64, 1 << 22, g)
    before = _trimmed_free()
    c = _call("f32", rv.RVSP_CUDA_ALGO_EXACT, A, B, T.float32)
    assert c[1].numel() > 400_000_000
    _release("f32", c)
    T.cuda.synchronize()
    other = T.empty(before - (2 << 30), dtype=T.uint8, device="cuda")
    del other
    T.cuda.empty_cache()
    kept = before - _trimmed_free()
    assert kept < 1 << 30, kept
    print("same", kept)


def _child(case, mb):
    import rvsp_b200 as rv
    import torch as T

    g = T.Generator(device="cuda")
    g.manual_seed(3)
    if case == "kept":
        return _kept(g)
    fn, algo = "f32", rv.RVSP_CUDA_ALGO_EXACT
    if case == "oneshot":  # 410 MB of slots, 410 of C
        A, B = _strata(200000, 16, 65536, g), _strata(65536, 16, 65536, g)
    if case == "f64":  # 1230 MB of slots, 440 of C
        fn = "f64"
        A, B = _strata(200000, 32, 65536, g), _strata(65536, 16, 192, g)
    if case == "slots_learned":  # 1.1 GB of loose slots, 0.8 of tight ones, 0.5 of C
        A, B = _strata(150000, 30, 235, g), _strata(160000, 30, 265, g)
        A[3].add_(T.arange(150000, device="cuda", dtype=T.int32).repeat_interleave(30))
        B[3].add_(T.arange(160000, device="cuda", dtype=T.int32).repeat_interleave(30))
        A, B = (150000, 160000) + A[2:], (160000, 161000) + B[2:]
        algo = rv.RVSP_CUDA_ALGO_LEARNED
    if case.startswith("heavy"):  # 600 MB of segment lists and what builds them, 550 of C
        A, B = _strata(3000, 600, 204800, g), _strata(204800, 40, 1 << 18, g)
        algo = rv.RVSP_CUDA_ALGO_LEARNED if case == "heavy_learned" else algo
        fn = {"heavy_descriptor": "descriptor", "heavy_f64": "f64"}.get(case, fn)
    small = _strata(512, 4, 512, g)
    if fn == "f64":
        A, B, small = ((*M[:4], M[4].double()) for M in (A, B, small))
    vd = A[4].dtype
    _release(fn, _call(fn, algo, small, small, vd))  # the library and its kernels are loaded
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


@pytest.mark.parametrize("case,mb", [
    ("oneshot", 640), ("f64", 1200), ("f64", 1450), ("heavy_exact", 850), ("heavy_learned", 1600),
    ("slots_learned", 1700), ("heavy_descriptor", 900), ("heavy_f64", 2250)])
def test_little_memory(gpu_lib, case, mb):
    _run(case, mb)


def test_lists_are_not_kept(gpu_lib):
    _run("kept", 0)


def _run(case, mb):
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
