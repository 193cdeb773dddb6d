"""The table-driven logarithm of the curved-ray traveltime against log(), on the
CPU: the same source (csrc/logtab.cuh) compiled as C++.  The bound is derived from
the method: the polynomial's first neglected term z^7 / 7 with |z| <= 2^-7 + 2^-24
(2^-51.8), three roundings of values below 2^-6 and two of size |log x| + 0.7."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "logtab.cuh"
extern "C" void run(const double *x, double *y, long n) {
    using std::log; using std::fma;
    static pstm::LogEntry tab[pstm::kLogEntries];
    for (int i = 0; i < pstm::kLogEntries; ++i) tab[i] = pstm::log_entry(i);
    for (long i = 0; i < n; ++i) y[i] = pstm::log_by_table(tab, x[i]);
}
"""


def test_log_table_against_libm(tmp_path):
    src, lib = tmp_path / "logtab.cpp", tmp_path / "logtab.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "pstm_b200", "csrc"),
                    "-o", str(lib), str(src)], check=True)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]
    rng = np.random.default_rng(3)
    edges = (1.0 + np.arange(65) / 64.0)[:, None] * (1.0 + np.array([-2.0, -1.0, 0.0, 1.0, 2.0]) * 2.0 ** -52)
    x = np.concatenate([np.exp(rng.uniform(-14, 14, 400000)), 1.0 + rng.uniform(-1e-6, 1e-6, 20000),
                        rng.uniform(1.0, 2.0, 400000), edges.ravel(), [2.0 ** -1000, 2.0 ** 1000]])
    y = np.empty_like(x)
    f(x.ctypes.data, y.ctypes.data, len(x))
    ref = np.log(x.astype(np.longdouble))
    err = np.abs(y.astype(np.longdouble) - ref)
    assert np.all(err <= 2.0 ** -50 + 2.0 ** -52 * np.abs(ref))


def test_log_table_is_left_with_roundings(tmp_path):
    """No truncation error beside the roundings of a log(): z^7 / 7 with |z| <= 2^-8 +
    2^-24 is below 2^-58; the entry's rounding is 2^-54 (|log c| < 0.7), log 2's 2.3e-17
    per power of 2, and three sums of size |log x| + 2^-8 round by half a unit each:
    2^-53 (0.5 + 0.21 (1 + 1.45 |log x|) + 3 |log x| + 0.04) in all."""
    src, lib = tmp_path / "logtab.cpp", tmp_path / "logtab.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "pstm_b200", "csrc"),
                    "-o", str(lib), str(src)], check=True)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]
    edges = (1.0 + np.arange(257) / 256.0)[:, None] * (1.0 + np.array([-2.0, -1.0, 0.0, 1.0, 2.0]) * 2.0 ** -52)
    x = np.concatenate([np.exp(np.random.default_rng(4).uniform(-9, 9, 400000)), edges.ravel()])
    y = np.empty_like(x)
    f(x.ctypes.data, y.ctypes.data, len(x))
    ref = np.log(x.astype(np.longdouble))
    err = np.abs(y.astype(np.longdouble) - ref)
    assert np.all(err <= 2.0 ** -53 * (0.75 + 3.5 * np.abs(ref)))
