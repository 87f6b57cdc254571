"""The library's host code over a CUDA runtime without a GPU
(tests/cpp/fake_cudart.cpp): which kernels it launches, how, and what it
answers when a device refuses or a kernel reports.  Kernels do nothing."""
import ctypes as C
import glob
import os
import subprocess

import numpy as np

from psum_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class Launch(C.Structure):
    _fields_ = [("name", C.c_char * 256)] + [(k, C.c_int) for k in
                                             ("device", "grid", "block", "smem", "cooperative", "cluster", "captured")]


def build(path):
    """Link the library's objects with the fake runtime into `path`."""
    subprocess.run(["make", "-s", "-j8", "-C", os.path.join(ROOT, "psum_b200", "csrc")], check=True)
    objs = sorted(glob.glob(os.path.join(ROOT, "_build", "psum_b200", "*.o")))
    gomp = (glob.glob("/usr/lib/gcc/x86_64-linux-gnu/*/libgomp.so") + ["-lgomp"])[0]
    cmd = ["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-I/usr/local/cuda/include",
           os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), *objs, "-o", path, gomp]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(path)
    for name, (res, args) in _lib.PROTOTYPES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.fake_device_bytes.restype = C.c_ulonglong
    lib.fake_pinned.argtypes = [C.c_ulonglong, C.POINTER(C.c_void_p), C.c_int]
    return lib


class Fake:
    """One loaded fake library; `reset` puts the device back as a test expects it."""

    def __init__(self, path):
        self.lib = build(path)

    def reset(self):
        self.lib.fake_device(0, 148)
        self.lib.fake_refuse_cooperative(0)
        self.lib.fake_clear_log()

    def log(self):
        out = []
        for i in range(self.lib.fake_launches()):
            q = Launch()
            self.lib.fake_launch(i, C.byref(q))
            out.append(q)
        return out

    def kernels(self, part):
        """The launches so far of the kernels whose name contains `part`."""
        return [q for q in self.log() if part in q.name.decode()]

    def stream(self):
        s = C.c_void_p()
        assert self.lib.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
        return s

    def set_host_words(self, value):
        """Every pinned word that a kernel could report through."""
        out = (C.c_void_p * 64)()
        n = self.lib.fake_pinned(4096, out, 64)
        assert 0 < n <= 64
        for i in range(n):
            (C.c_int * 1024).from_address(out[i])[:] = [value] * 1024


def poisson(nodes, eps=None):
    """Five- or seven-point operator on a box with grounded faces, optionally with a coefficient per node (COO)."""
    n = int(np.prod(nodes))
    idx = np.arange(n).reshape(nodes)
    wall = np.ones(nodes, bool)
    wall[tuple(slice(1, -1) for _ in nodes)] = False
    e = np.ones(nodes) if eps is None else eps
    rows, cols, vals = [idx[wall]], [idx[wall]], [np.ones(wall.sum())]
    diag = np.zeros(nodes)
    inner = ~wall
    for a in range(len(nodes)):
        for d in (-1, 1):
            w = 0.5 * (e + np.roll(e, -d, axis=a))
            rows.append(idx[inner])
            cols.append(np.roll(idx, -d, axis=a)[inner])
            vals.append(-w[inner])
            diag += w
    rows.append(idx[inner])
    cols.append(idx[inner])
    vals.append(diag[inner])
    r, c, v = (np.concatenate(q) for q in (rows, cols, vals))
    return r.astype(np.uint64), c.astype(np.uint64), v


class Solver:
    def __init__(self, fake, kind, nodes, options="", eps=None):
        self.lib = fake.lib
        self.n = int(np.prod(nodes))
        self.h = C.c_void_p()
        assert self.lib.psum_mg_create(kind.encode(), C.byref(self.h)) == 0
        k = tuple(nodes) + (1,) * (3 - len(nodes))
        self.set_options(f"I {k[0]} J {k[1]} K {k[2]} depth 3 pre_relax 2 post_relax 2 max_cycles 4 correction_interval 2 " + options)
        r, c, v = poisson(nodes, eps)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        self.check(self.lib.psum_mg_set_matrix(self.h, self.n, self.n, r.size, p(r), p(c), p(v)))
        self.b, self.x = np.zeros(self.n), np.zeros(self.n)

    def set_options(self, options):
        self.check(self.lib.psum_mg_set_options(self.h, options.encode()))

    def set_source(self, idx, values, replace=False):
        idx, values = np.ascontiguousarray(idx, np.uint64), np.ascontiguousarray(values, np.float64)
        f = self.lib.psum_mg_set_source_replace if replace else self.lib.psum_mg_set_source_addback
        self.check(f(self.h, idx.size, idx.ctypes.data, values.ctypes.data))

    def check(self, code):
        assert code == 0, (code, self.lib.psum_last_error())

    def solve_async(self, stream=None):
        return self.lib.psum_mg_solve_async(self.h, self.b.ctypes.data, self.x.ctypes.data, stream)

    def solve(self):
        return self.lib.psum_mg_solve(self.h, self.b.ctypes.data, self.x.ctypes.data)

    def last_stats(self):
        i, d = C.c_int(), C.c_double()
        return self.lib.psum_mg_last_stats(self.h, C.byref(i), C.byref(i), C.byref(d), C.byref(d))

    def close(self):
        self.lib.psum_mg_destroy(self.h)


def step_context(fake, cells, n=1000, options="sort_interval 1"):
    """A particle context with one species; returns a function that runs one step with a solver, and one to close it."""
    lib, dim = fake.lib, len(cells)
    g = _lib.GridDesc()
    g.dim = dim
    for a in range(3):
        g.cells[a] = cells[a] if a < dim else 1
        g.lower[a], g.upper[a], g.periodic[a] = 0.0, float(g.cells[a]), 0
    ctx = C.c_void_p()
    assert lib.psum_pic_create(C.byref(g), 0, C.byref(ctx)) == 0
    assert lib.psum_pic_set_options(ctx, options.encode()) == 0
    sid = C.c_int()
    assert lib.psum_pic_add_species(ctx, C.byref(_lib.SpeciesDesc(1.0, 1.0, 1.0)), n, C.byref(sid)) == 0
    pos, vel = np.full((dim, n), 0.5), np.zeros((3, n))
    assert lib.psum_pic_load(ctx, sid.value, n, pos.ctypes.data, vel.ctypes.data) == 0
    assert lib.psum_pic_sort(ctx) == 0 and lib.psum_pic_deposit(ctx) == 0

    def step(solver):
        return lib.psum_pic_step(ctx, solver.h, 0.0, solver.b.ctypes.data, solver.x.ctypes.data, 0.1, 0, (C.c_double * 3)())
    return step, lambda: lib.psum_pic_destroy(ctx)
