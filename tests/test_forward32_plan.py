"""The FP32 forward kernel's shared memory: whatever a problem's batch mates are, the form that it
runs in lies within the bytes that the launch allocates, and its threads hold its states."""

import ctypes as C
import os
import subprocess

import pytest

from argweaver_gb300 import build

STATES = [1, 2, 31, 32, 33, 99, 192, 193, 383, 384, 385, 512, 513, 767, 768, 769, 930, 1024, 1025, 1152,
          1153, 1491, 1535, 1536, 1537, 2047, 2048, 2049, 2580, 3071, 3072]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("f32") / "libf32.so")
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + build.INCLUDE,
                    "-I" + build.CSRC, "-I/usr/local/cuda/include", "-o", out,
                    os.path.join(here, "forward32_plan_shim.cpp")], check=True)
    return C.CDLL(out)


def _shapes(times):
    """Largest trees of up to 3,072 states: row entries from one a state to a node of every time."""
    for s in STATES:
        for share in (1, 3, 6, 13, 18, 23, times - 1):
            for nodes in (1, 63, 457, 1023):
                yield s, s * min(share, s, times - 1), nodes


@pytest.mark.parametrize("times", [4, 21, 22, 32])
def test_every_form_fits_its_launch(lib, times):
    smem, form = C.c_int(0), (C.c_int * 4)()
    shapes = list(_shapes(times))
    mates = [m for m in shapes if m[2] in (1, 1023)]
    for z in shapes:
        for b in [z] + mates[::5]:
            big = [max(x, y) for x, y in zip(z, b)]
            for least in (1, 2, 4, 8):
                need = lib.plan_bytes(*z, *big, int(times > 21), least, C.byref(smem), form)
                assert need <= smem.value <= 222 * 1024, (z, big, least, list(form))
                kpt, bufs, staged, owners = form
                wide = big[0] > 4 * 384
                assert owners <= (512 if wide else 384) and kpt * owners >= z[0]
                assert kpt in (1, 2, 3, 4, 8) and not (kpt <= 2 and not staged)
                if kpt == 3:
                    assert big[0] > 768  # only in the kernels for larger batches


def test_long_nodes_beside_small_problems(lib):
    """Rows of a large batch mate do not move a small problem's arrays: 100 haplotypes of 32 time
    points at N = 1e6 beside 99 and 384 states, and at their own size."""
    smem, form = C.c_int(0), (C.c_int * 4)()
    for s, m, n in ((99, 594, 15), (384, 2600, 95)):
        need = lib.plan_bytes(s, m, n, 2580, 53212, 197, 1, 1, C.byref(smem), form)
        assert need <= smem.value and list(form)[:3] == [1, 1, 1]
        alone = lib.plan_bytes(s, m, n, s, m, n, 1, 1, C.byref(smem), form)
        assert alone == need
