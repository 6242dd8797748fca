"""The library's host code on a stand-in for the CUDA runtime
(tests/cpp/fake_cudart.cpp), for tests without a GPU: which kernels a call
launches, what it does when a launch or an allocation fails, and what memory it
holds. Kernels do not run, so no value that one would compute is checked here."""
import ctypes as ct
import os
import subprocess

import numpy as np

from conftest import ROOT

OK, ERR_CUDA, ERR_NOMEM = 0, 3, 4
_vp, _d = ct.c_void_p, ct.c_double


def build(out_dir):
    """Links the library's object files with the stand-in; returns the path."""
    objs = os.path.join(ROOT, "mcpi_b200", "_build")
    subprocess.run(["make", "-s", "-j8", "-C", os.path.join(ROOT, "mcpi_b200")], check=True)
    so = os.path.join(str(out_dir), "libmcpi_fake.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include", "-o", so,
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"),
                    *sorted(os.path.join(objs, o) for o in os.listdir(objs) if o.endswith(".o")),
                    "-Wl,-Bsymbolic", "-Wl,--no-undefined"], check=True)
    return so


class Fake:
    def __init__(self, so):
        self.L = L = ct.CDLL(so)
        L.fake_log.restype = ct.c_char_p
        L.mcpi_last_error.restype = ct.c_char_p
        for f in ("fake_pool_held", "fake_used", "fake_synced_log"):
            getattr(L, f).restype = ct.c_size_t
        L.fake_headroom.restype = None
        L.fake_headroom.argtypes = [ct.c_size_t]
        L.fake_fail_launch.argtypes = [ct.c_long]
        L.fake_fail_pool.argtypes = [ct.c_long, ct.c_int]

    def reset(self):
        self.L.fake_reset()

    def kernels(self, call):
        """Names (mangled) of the kernels that call() launches; its return value has to be OK."""
        self.L.fake_clear_log()
        assert call() == OK, self.L.mcpi_last_error()
        return self.L.fake_log().decode().split()

    def unfinished(self, call):
        """Names of the kernels launched by call() that the host has not waited for at its end."""
        self.L.fake_clear_log()
        assert call() == OK, self.L.mcpi_last_error()
        return self.L.fake_log()[self.L.fake_synced_log():].decode().split()

    def space(self, N, M):
        return Space(self, N, M)

    def batch(self, members, lm, integrals):
        return Batch(self, members, lm, integrals)


def _ptr(a):
    return a.ctypes.data_as(_vp)


class Space:
    """A space whose device pointers are numpy arrays (the stand-in's device memory is host memory)."""

    def __init__(self, fake, N, M):
        self.fake, self.L, self.N, self.M = fake, fake.L, N, M
        self.h = _vp()
        assert self.L.mcpi_space_create(N, M, 0, ct.byref(self.h)) == OK
        nc = ct.c_int64()
        self.L.mcpi_nc(N, M, ct.byref(nc))
        self.nc = nc.value
        self.x, self.y = np.zeros(self.nc, np.complex128), np.zeros(self.nc, np.complex128)

    def option(self, opt, value):
        assert self.L.mcpi_space_set_option(self.h, opt, value) == OK

    def set_integrals(self, Ho, Hint):
        self.Ho = np.ascontiguousarray(Ho, np.complex128)
        self.Hint = np.ascontiguousarray(Hint, np.complex128)
        return self.L.mcpi_set_integrals(self.h, _ptr(self.Ho), _ptr(self.Hint), 0)

    def apply_h(self):
        return self.L.mcpi_apply_h(self.h, _ptr(self.x), _ptr(self.y))

    def apply_h_adjoint(self):
        return self.L.mcpi_apply_h_adjoint(self.h, _ptr(self.x), _ptr(self.y))

    def rows(self, r0, r1, entry="mcpi_apply_h_rows"):
        return getattr(self.L, entry)(self.h, _ptr(self.x), ct.c_int64(r0), ct.c_int64(r1), _ptr(self.y))

    def density(self, order, same=True):
        self.rho = np.zeros(self.M ** (2 * order), np.complex128)
        phi = self.x if same else self.y
        name = ("mcpi_rho%d" if same else "mcpi_trans_rho%d") % order
        args = (_ptr(phi), _ptr(self.rho)) if same else (_ptr(phi), _ptr(self.x), _ptr(self.rho))
        return getattr(self.L, name)(self.h, *args)

    def dot(self):
        return self.L.mcpi_dot(self.h, _ptr(self.x), _ptr(self.y), _ptr(np.zeros(2)))

    def lanczos(self, lm):
        if getattr(self, "V", None) is None or self.V.shape[0] != lm:
            self.V = np.zeros((lm, self.nc), np.complex128)
        return self.L.mcpi_lanczos(self.h, _ptr(self.V), lm, _ptr(np.zeros(2 * lm)), _ptr(np.zeros(lm)),
                                   ct.byref(ct.c_int()))

    def ground(self, lm, lowmem=False):
        f = self.L.mcpi_ground_lowmem if lowmem else self.L.mcpi_ground
        return f(self.h, _ptr(self.x), lm, ct.byref(_d()), ct.byref(ct.c_int()))

    def close(self):
        self.L.mcpi_space_destroy(self.h)


class Batch:
    def __init__(self, fake, members, lm, integrals):
        self.L, self.n, self.h = fake.L, len(members), _vp()
        N, M = (np.array(x, np.int32) for x in zip(*members))
        self.rc = self.L.mcpi_batch_create(self.n, _ptr(N), _ptr(M), lm, 0, ct.byref(self.h))
        for k, m in enumerate(M if self.rc == OK else []):
            Ho, Hint = (np.ascontiguousarray(a, np.complex128) for a in integrals(int(m), 1.0))
            assert self.L.mcpi_batch_set_integrals(self.h, k, _ptr(Ho), _ptr(Hint), 0) == OK
            nc = ct.c_int64()
            assert self.L.mcpi_batch_member_size(self.h, k, ct.byref(nc)) == OK
            assert self.L.mcpi_batch_set_start(self.h, k, _ptr(np.zeros(nc.value, np.complex128))) == OK

    def run(self):
        return self.L.mcpi_batch_run(self.h, _ptr(np.zeros(self.n)), _ptr(np.zeros(self.n, np.int32)))

    def close(self):
        if self.h:
            self.L.mcpi_batch_destroy(self.h)
