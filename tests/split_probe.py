"""Compiles tests/native/split_probe.cu for the GPU tests of a single split."""
import ctypes
import os
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))


def load(folder):
    """The probe library, built in ``folder`` with the flags of the package."""
    from oqupy_gb300 import build
    so = os.path.join(str(folder), "split_probe.so")
    subprocess.run([build.nvcc()] + build.FLAGS + build.ARCH
                   + ["-shared", os.path.join(HERE, "native", "split_probe.cu"), "-o", so, "-lcudart"], check=True)
    return ctypes.CDLL(so)


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def split(lib, A, epsrel, precision="complex128", qr_cut=0.0):
    """``(U, s, V)`` of the kept part of A (R x N, R >= N), A ~ U diag(s) V^H,
    and the status; the factor that the split does not return is formed here."""
    A = np.asarray(A, dtype=np.complex128)
    R, N = A.shape
    a = np.ascontiguousarray(A.T)
    W = np.zeros(R * N, dtype=np.complex128)
    s, meta = np.zeros(N), np.zeros(4, dtype=np.int32)
    rc = lib.split_probe(int(precision == "mixed"), _p(a), R, N, ctypes.c_double(epsrel), ctypes.c_double(qr_cut),
                         _p(W), _p(s), _p(meta))
    assert rc == 0, rc
    kk, flip, status = (int(x) for x in meta[:3])
    ld = N if flip else R
    W, s = W[:ld * kk].reshape(kk, ld).T, s[:kk]
    with np.errstate(all="ignore"):
        if flip:                                   # W = A^H U Sigma
            V = W / s
            U = (A / s[0]) @ V / (s / s[0])
        else:                                      # W = A V Sigma
            U = W / s
            V = (A / s[0]).conj().T @ U / (s / s[0])
    return U, s, V, status


def rsqrt(lib, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    d, f = np.empty_like(x), np.empty_like(x)
    assert lib.rsqrt_probe(_p(x), _p(d), _p(f), len(x)) == 0
    return d, f
