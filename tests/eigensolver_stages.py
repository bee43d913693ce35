"""Builds and calls tests/native/eigensolver_stages.cu."""
import ctypes
import os
import subprocess

import numpy as np

from wanniernlqg_b200 import build

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "eigensolver_stages.cu")
LIB = os.path.join(os.path.dirname(SOURCE), "_build", "libeigensolver_stages.so")


def load():
    depends = [SOURCE] + build.DEPENDS
    if not os.path.exists(LIB) or any(os.path.getmtime(f) > os.path.getmtime(LIB) for f in depends):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
                        "-shared", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-I",
                        os.path.join(build.HERE, "csrc"), "-o", LIB + ".tmp", SOURCE, "-lcudart"], check=True)
        os.replace(LIB + ".tmp", LIB)
    return ctypes.CDLL(LIB).eigensolver_stages


def run(stages, h, *, chains=1, warm=True, start=None):
    """Stage 1's vectors V [n, np, np] (or ``start`` in their place), stage 2's E [n, nw] and U [n, nw, nw]
    of the Hermitian h [n, nw, nw], whose points form ``chains`` runs of warm-started neighbours."""
    n, nw = h.shape[:2]
    m = nw + nw % 2
    hc = np.ascontiguousarray(h.transpose(0, 2, 1))
    v = np.zeros((n, m, m), np.complex64)
    if start is not None:
        v[:, np.arange(m), np.arange(m)] = 1.0
        v[:, :nw, :nw] = start.transpose(0, 2, 1)
    e, u = np.zeros((n, nw)), np.zeros((n, nw, nw), np.complex128)
    p = [ctypes.c_void_p(x.ctypes.data) for x in (hc, v, e, u)]
    code = stages(p[0], ctypes.c_int64(n), nw, ctypes.c_int64(chains), int(warm), int(start is not None), p[1], p[2], p[3])
    assert code == 0, f"CUDA error {code}"
    return v.transpose(0, 2, 1), e, u.transpose(0, 2, 1)
