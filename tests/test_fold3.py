"""fold3_add_long (master-of-puppets_b200/csrc/fold.h), three interleaved folds, equals the
plain serial loop bit for bit: screen-like edge values and slopes, coarse grids (ties), half-ulp
slopes, zero crossings, subnormal, infinite and NaN values; counts from 17 (its smallest) up."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("fold3") / "fold3_check.so"
    subprocess.run(["gcc", "-O2", "-std=c11", "-shared", "-fPIC", "-ffp-contract=off",
                    "-I", str(ROOT / "master-of-puppets_b200" / "csrc"),
                    str(ROOT / "tests" / "native" / "fold3_check.c"), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    L.fold3_check.argtypes = [C.c_int] + [C.c_void_p] * 4
    return L


@pytest.mark.parametrize("kind", ["screen", "grid", "half_ulp", "tiny", "special"])
def test_fold3_matches_serial(lib, kind):
    rng = np.random.default_rng(len(kind))
    n = 60000
    w = rng.uniform(-1, 1, 3 * n) * 2.0 ** rng.integers(-6, 22, 3 * n)
    d = rng.uniform(-1, 1, 3 * n) * 2.0 ** rng.integers(-12, 12, 3 * n)
    if kind == "grid":
        w, d = np.round(w * 8) / 8, np.round(d * 64) / 64
    w, d = w.astype(np.float32), d.astype(np.float32)
    if kind == "half_ulp":
        d = (np.spacing(w) * (rng.integers(-9, 9, 3 * n) + 0.5)).astype(np.float32)
    elif kind == "tiny":
        w = (w * np.float32(2.0 ** -130)).astype(np.float32)
        d = (d * np.float32(2.0 ** -135)).astype(np.float32)
    elif kind == "special":
        sp = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e38, -1e38, 1e-45], np.float32)
        w[::2] = sp[rng.integers(0, 8, w[::2].size)]
        d[1::3] = sp[rng.integers(0, 8, d[1::3].size)]
    k = rng.integers(17, 3000 if kind != "screen" else 9000, n).astype(np.int32)
    k[:200] = np.arange(17, 217)
    bad = C.c_int(-1)
    fails = lib.fold3_check(n, w.ctypes.data, d.ctypes.data, k.ctypes.data, C.byref(bad))
    i = bad.value
    assert fails == 0, (fails, w[3 * i:3 * i + 3], d[3 * i:3 * i + 3], k[i])
