"""The library's calls work again after the device's primary context has been reset (what cudaDeviceReset does):
nothing that it remembers of the old context is taken for the new one's."""
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = textwrap.dedent("""
    import ctypes
    import numpy as np
    from scalingelections_b200 import _lib

    cu = ctypes.CDLL("libcuda.so.1")
    L = _lib.lib()

    def ok(code):
        assert code == 0, code

    ok(cu.cuInit(0))

    def alloc(n):
        p = ctypes.c_uint64()
        ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(n)))
        return p.value

    results = []
    for turn in range(2):
        ctx = ctypes.c_void_p()
        ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(ctx), 0))
        ok(cu.cuCtxSetCurrent(ctx))
        got = []
        for C, mode in ((300, 0), (300, 1), (1000, 0), (1000, 5), (1700, 0)):
            d = np.random.default_rng(C).integers(0, 9000, size=(C, C)).astype(np.uint32)
            nbytes = L.se_closure_workspace_bytes_flow(C, 16, 0)
            a, b, w = alloc(d.nbytes), alloc(d.nbytes), alloc(nbytes)
            ok(cu.cuMemcpyHtoD_v2(ctypes.c_uint64(a), d.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(d.nbytes)))
            _lib.check(L.se_closure_set_mode(mode))
            _lib.check(L.se_closure(a, C, C, b, C, 16, 0, w, nbytes, None))
            out = np.empty_like(d)
            ok(cu.cuMemcpyDtoH_v2(out.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(b), ctypes.c_size_t(d.nbytes)))
            got.append(out)
        results.append(got)
        ok(cu.cuCtxSynchronize())
        ok(cu.cuDevicePrimaryCtxReset_v2(0))
    assert all(np.array_equal(x, y) for x, y in zip(*results))
    assert np.array_equal(results[0][0], results[0][1])
    print("done")
""")


def test_closures_after_a_reset():
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parent.parent)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]
