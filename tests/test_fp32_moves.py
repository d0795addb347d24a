"""Switch moves as the FP32 steps read them: a complement of 1 without a sign for probabilities of
1/2 and more (those that round above 1 among them), the negated probability below."""

import ctypes as C
import os
import subprocess

import numpy as np

from argweaver_gb300 import build


def test_moves(tmp_path):
    src, out = tmp_path / "moves.cpp", str(tmp_path / "libmoves.so")
    src.write_text('#include "awg_internal.h"\nextern "C" float move_of(double p) { return awg::fp32_move(p); }\n')
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + build.INCLUDE,
                    "-I" + build.CSRC, "-I/usr/local/cuda/include", "-o", out, str(src)], check=True)
    f = C.CDLL(out).move_of
    f.restype, f.argtypes = C.c_float, [C.c_double]
    for p in (1.0, 1.0 + 2.0 ** -52, 1.0 + 1e-12, 1.0 - 2.0 ** -53, 1.0 - 1e-9, 0.75, 0.5):
        m = np.float32(f(p))
        assert not np.signbit(m) and m == np.float32(max(1.0 - p, 0.0))
    for p in (0.0, 1e-300, 1e-20, 0.25, np.nextafter(0.5, 0)):
        m = np.float32(f(p))
        assert np.signbit(m) and -m == np.float32(p)
