"""The library's host code on the fake runtime of fake_cudart.cpp: which kernels a call launches,
in which order it uses and releases buffers, and what it does when a call fails (no GPU)."""
import ctypes
import importlib.util
import os
import re
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "randlinearalgebra.jl_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

LEFT, RIGHT = 0, 1
F32, F64 = 0, 1
KINDS = {"sparse_sign": 0, "count_sketch": 1, "srht": 2, "fjlt": 3, "gaussian": 4}
vp, i64 = ctypes.c_void_p, ctypes.c_int64
BASE = 1 << 40  # stands for the address of an operand: never read


def build(folder):
    """The objects of the library (compiled when out of date) linked with the fake runtime (its own
    calls bind to it also when a real runtime is loaded); calls that it does not have end the process."""
    spec = importlib.util.spec_from_file_location("rla_build", os.path.join(PKG, "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    os.makedirs(b.OBJ, exist_ok=True)
    with ThreadPoolExecutor(8) as ex:
        objs = list(ex.map(lambda src: b._compile(src, False, False, False), b._sources()))
    fake, stubs = os.path.join(folder, "fake.o"), os.path.join(folder, "stubs.c")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-I", os.path.join(CUDA, "include"), "-c",
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", fake], check=True)
    nm = lambda args: subprocess.run(["nm", *args], check=True, capture_output=True, text=True).stdout
    need = set(re.findall(r" U ((?:__)?cu(?:da)?[A-Z]\w+)$", nm(objs), re.M))
    have = set(re.findall(r" T (\w+)$", nm([fake]), re.M))
    with open(stubs, "w") as f:
        f.write("#include <stdio.h>\n#include <stdlib.h>\n")
        for n in sorted(need - have):
            f.write('void %s(void) { fprintf(stderr, "fake runtime: %s\\n"); abort(); }\n' % (n, n))
    lib = os.path.join(folder, "librla_fake.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-o", lib, *objs, fake, "-x", "c", stubs], check=True)
    return lib


class Params(ctypes.Structure):
    _fields_ = [("kind", ctypes.c_int), ("card", ctypes.c_int), ("dtype", ctypes.c_int), ("compression_dim", i64),
                ("long_dim", i64), ("nnz", i64), ("block_size", i64), ("sparsity", ctypes.c_double),
                ("seed", ctypes.c_uint64)]


class Fake:
    def __init__(self, path):
        self.path = path
        self.lib = ctypes.CDLL(path)
        self.lib.fake_log.restype = ctypes.c_char_p
        self.lib.rla_ctx_last_error.restype = ctypes.c_char_p

    def fresh(self, folder):
        """Another instance of the library, with none of this one's state."""
        return Fake(shutil.copy(self.path, os.path.join(str(folder), "librla_fake_fresh.so")))

    def reset(self):
        self.lib.fake_reset()

    def log(self):
        return self.lib.fake_log().decode().splitlines()

    def fail_after(self, call, ok):
        self.lib.fake_fail_after(call.encode(), ok)

    def capturing(self, on):
        self.lib.fake_capturing(int(on))

    def context(self):
        ctx = vp()
        assert self.lib.rla_ctx_create(0, None, ctypes.byref(ctx)) == 0
        return ctx

    def create(self, ctx, kind, s, L, card=LEFT, dtype=F32, nnz=1):
        """(status, sketch)"""
        sk = vp()
        p = Params(KINDS[kind], card, dtype, s, L, nnz, 10, 0.0, 7)
        return self.lib.rla_sketch_create(ctx, ctypes.byref(p), ctypes.byref(sk)), sk

    def sketch(self, ctx, *a, **k):
        rc, sk = self.create(ctx, *a, **k)
        assert rc == 0, self.lib.rla_ctx_last_error(ctx)
        return sk

    def mul(self, ctx, sk, kind_shape, card, adjoint=False, row_a=False, row_c=False, beta=0.0, pad=0, a=BASE, c=2 * BASE,
            wait=True):
        """mul!(C, S, A) (Left) / mul!(C, A, S) (Right) or with S': shape (s, L, nv)."""
        s, L, nv = kind_shape
        long_, short = ((L, nv), (s, nv)) if card == LEFT else ((nv, L), (nv, s))
        A, C = (short, long_) if adjoint else (long_, short)
        lda, ldc = (A[1] if row_a else A[0]) + pad, (C[1] if row_c else C[0]) + pad
        fn = self.lib.rla_sketch_mul if wait else self.lib.rla_sketch_mul_async
        fn.argtypes = [vp, vp, ctypes.c_int, ctypes.c_int, i64, i64, vp, i64, ctypes.c_int, i64, i64, vp, i64, ctypes.c_int,
                       ctypes.c_double, ctypes.c_double]
        return fn(ctx, sk, 0 if card == LEFT else 1, int(adjoint), C[0], C[1], c, ldc, int(row_c), A[0], A[1], a, lda,
                  int(row_a), 1.0, beta)

    def launches(self):
        """Names of the kernels launched since the last reset, in order."""
        return [ln.split()[1] for ln in self.log() if ln.startswith("launch ")]


_fake = []


@pytest.fixture
def fake(tmp_path_factory):
    if not _fake:
        _fake.append(Fake(build(str(tmp_path_factory.mktemp("fake_cuda")))))
    _fake[0].reset()
    yield _fake[0]
    _fake[0].reset()
