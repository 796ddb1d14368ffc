"""An allocation that fails in the middle of a count leaves the context fit for
the next one: no freed buffer is used or freed again, and no catalogue passes
for sorted whose sorted arrays were replaced.  The host layer (ctx.c, bins.c) is
compiled against a runtime on the host (fake_cuda.c) that fails the k-th
allocation and checks what each launch is given; no GPU is involved."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fcfc_gb300 import build, capi

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fcfc_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.check_call(
        ["gcc", "-O1", "-std=gnu11", "-ffp-contract=off", "-shared", "-fPIC",
         "-Wl,-Bsymbolic",       # (a loaded libcudart takes no calls)
         "-I", CSRC, "-I", os.path.join(build.cuda_home(), "include"), "-o", so,
         os.path.join(HERE, "fake_cuda.c")] +
        [os.path.join(CSRC, f) for f in ("ctx.c", "bins.c")] + ["-lm"])
    lib = C.CDLL(so)
    for name, (res, args) in capi.PROTOTYPES.items():
        if hasattr(lib, name):
            getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    lib.fake_what.restype = C.c_char_p
    return lib


class Ctx:
    def __init__(self, lib):
        self.lib, self.keep = lib, []
        b, keep = capi.make_binning(capi.GEOM_BOX, 1, box=1000.0, smin=0,
                                    smax=20, ds=2, nmu=10)
        self.h = C.c_void_p()
        assert lib.fcfcg_create(C.byref(b), 0, C.byref(self.h)) == 0
        self.out = np.zeros(100, np.int64)

    def load(self, slot, n):
        x = np.random.default_rng(n).random((3, n)) * 1000.0
        self.keep.append(x)
        return self.lib.fcfcg_load_catalog(self.h, slot, n, *map(capi.ptr, x),
                                           None)

    def count(self, a, b):
        return self.lib.fcfcg_count(self.h, a, b, int(a == b), 0, 0,
                                    capi.ptr(self.out), None)

    def batch(self, sizes):
        jobs = (capi.Job * len(sizes))()
        for j, n in zip(jobs, sizes):
            x = np.random.default_rng(n).random((3, n)) * 900.0
            out = np.zeros(100, np.int64)
            self.keep += [x, out]
            j.n = n
            j.x, j.y, j.z = (c.ctypes.data_as(capi._dp) for c in x)
            j.box = (C.c_double * 3)(900.0, 900.0, 900.0)
            j.icnt = out.ctypes.data_as(C.POINTER(C.c_int64))
        rc = self.lib.fcfcg_count_batch(self.h, jobs, len(sizes), 0, 0, 0)
        assert rc or not any(j.status for j in jobs)
        return rc

    def close(self):
        self.lib.fcfcg_destroy(self.h)


def _fails_then_works(lib, first, call, after):
    """call with its k-th allocation failing, k = 1, 2, ... until none fails."""
    lib.fake_reset()
    for k in range(1, 100):
        c = Ctx(lib)
        first(c)
        lib.fake_fail_at(k)
        rc = call(c)
        armed = lib.fake_armed()
        lib.fake_fail_at(0)
        for f in after:
            assert f(c) == 0, k
            assert lib.fake_faults() == 0, (k, lib.fake_what())
        c.close()
        assert lib.fake_faults() == 0, (k, lib.fake_what())
        if armed:                        # fewer allocations than k
            assert rc == 0 and k > 1
            return
        assert rc != 0
    raise AssertionError("never ran through")


@pytest.mark.parametrize("then", [30000, 900])
def test_count_after_failed_count(lib, then):
    """The sorted arrays of a catalogue that grew, then of the same or of one
    that fits what was allocated first."""
    def first(c):
        assert c.load(0, 30000) == 0
        assert c.load(0, 1000) == 0 and c.count(0, 0) == 0
        assert c.load(0, 30000) == 0
    _fails_then_works(lib, first, lambda c: c.count(0, 0),
                      [lambda c: c.load(0, then), lambda c: c.count(0, 0)])


def test_count_in_the_old_grid_after_failed_count(lib):
    """A cross count in a finer grid replaces the blocks of a sorted catalogue
    and fails; the catalogue is counted alone, in the grid it was sorted for."""
    def first(c):
        assert c.load(0, 2000) == 0 and c.count(0, 0) == 0
        assert c.load(1, 2000000) == 0
    _fails_then_works(lib, first, lambda c: c.count(1, 0),
                      [lambda c: c.count(0, 0), lambda c: c.count(1, 0)])


def test_batch_after_failed_batch(lib):
    def first(c):
        assert c.batch([500, 600]) == 0
    _fails_then_works(lib, first, lambda c: c.batch([30000, 40000, 900]),
                      [lambda c: c.batch([500, 600]),
                       lambda c: c.batch([30000, 40000, 900])])
