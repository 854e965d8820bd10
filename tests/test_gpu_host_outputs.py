"""The host calls write nothing past the caller's output arrays: each array ends
at a page that must not be touched, so a copy that runs over ends the process."""
import ctypes as C
import mmap
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class Guarded:
    """count doubles that end where an inaccessible page begins."""

    def __init__(self, count):
        page = mmap.PAGESIZE
        size = -(-count * 8 // page) * page
        self.map = mmap.mmap(-1, size + page)
        base = C.addressof(C.c_char.from_buffer(self.map))
        libc = C.CDLL(None, use_errno=True)
        libc.mprotect.argtypes = [C.c_void_p, C.c_size_t, C.c_int]
        assert libc.mprotect(base + size, page, 0) == 0
        self.ptr = C.c_void_p(base + size - count * 8)
        self.array = np.frombuffer((C.c_char * (count * 8)).from_address(self.ptr.value), dtype=np.float64)


def check(variant, t):
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(130, 1111, t, wXL=3, seed=5, hsig_uniform=True)
    nt = t if variant == "eigen" else 1
    with Engine(pb.n, 3, 1, t, 256, variant=variant) as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)
        XR = np.asfortranarray(pb.XR)
        x = C.c_void_p(XR.ctypes.data)
        B0, SE0, P0 = e.run_snps_compact(XR)
        B, SE, P = (Guarded(nt * pb.m * 4) for _ in range(3))
        assert e.L.fglsgpu_run_snps_compact(e.handle, x, pb.m, B.ptr, SE.ptr, P.ptr) == 0
        for got, want in ((B, B0), (SE, SE0), (P, P0)):
            assert np.array_equal(got.array, want.ravel())
        B, V = Guarded(nt * pb.m * 4), Guarded(nt * pb.m * 16)
        assert e.L.fglsgpu_run_snps(e.handle, x, pb.m, B.ptr, V.ptr) == 0
        assert np.array_equal(B.array, B0.ravel())


@pytest.mark.parametrize("variant,t", [("chol", 1), ("eigen", 1), ("eigen", 3)])
def test_outputs_end_at_the_caller_arrays(variant, t):
    code = (f"import sys; sys.path[:0] = [{os.path.join(ROOT, 'cugwas-proto_gb300')!r}, {os.path.dirname(__file__)!r}]\n"
            f"import test_gpu_host_outputs as t\nt.check({variant!r}, {t})\nprint('ok')\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0 and "ok" in r.stdout, (r.returncode, r.stderr[-500:])
