"""div_const (master-of-puppets_b200/csrc/fold.h) gives the division's results where the kernels
use it: an angle over 2 pi or pi plus 0.5, for every finite float, and a byte over 255."""
import concurrent.futures
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("div") / "div_const_check.so"
    cmd = ["gcc", "-O3", "-std=c11", "-shared", "-fPIC", "-ffp-contract=off",
           "-I", str(ROOT / "master-of-puppets_b200" / "csrc"),
           str(ROOT / "tests" / "native" / "div_const_check.c"), "-o", str(so), "-lm"]
    if " fma " in Path("/proc/cpuinfo").read_text():  # fmaf as an instruction, not a call
        cmd += ["-mfma", "-mavx2"]
    subprocess.run(cmd, check=True)
    L = C.CDLL(str(so))
    L.div_const_angles.argtypes = [C.c_uint64, C.c_uint64, C.c_int, C.c_void_p]
    L.div_const_angles.restype = C.c_long
    return L


@pytest.mark.parametrize("two", [0, 1])
def test_every_angle(lib, two):
    step = 1 << 28
    bad = [C.c_uint32() for _ in range(16)]
    with concurrent.futures.ThreadPoolExecutor(os.cpu_count()) as ex:  # ctypes drops the GIL
        n = list(ex.map(lambda k: lib.div_const_angles(k * step, (k + 1) * step, two,
                                                       C.byref(bad[k])), range(16)))
    assert sum(n) == 0, [(c, hex(b.value)) for c, b in zip(n, bad) if c]


def test_every_byte(lib):
    assert lib.div_const_bytes() == 0
