"""The folds as the device computes them (master-of-puppets_b200/csrc/fold.h): its approximate
division, which the host build of the header does not have, never lets a jump pass its binade's
edge, and the results are the serial loop's bit for bit."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("fold") / "fold_gpu.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-fmad=false", "-prec-div=true", "-ftz=false", "-shared", "-Xcompiler", "-fPIC",
                    "-cudart", "shared", "-I", str(ROOT / "master-of-puppets_b200" / "csrc"),
                    str(ROOT / "tests" / "native" / "fold_gpu.cu"), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    L.launch_folds.argtypes = [C.c_int] + [C.c_void_p] * 4
    L.launch_rooms.argtypes = [C.c_int] + [C.c_void_p] * 3
    return L


def _run(launch, *arrays):
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]
    bad = torch.zeros(2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    launch(arrays[-1].size, *(t.data_ptr() for t in dev), bad.data_ptr())
    torch.cuda.synchronize()
    return bad.tolist()


def test_rooms(lib):
    rng = np.random.default_rng(1)
    top = (1 << 24) - 1
    den = np.concatenate([np.full(top + 1, 1), np.repeat([2, 3, 5, 7, 4097, top], 100000),
                          (2.0 ** rng.uniform(0.0, 24.0, 4000000)).astype(np.int64).clip(1, top)])
    num = np.concatenate([np.arange(top + 1), rng.integers(0, top + 1, den.size - top - 1)])
    exact = rng.random(den.size) < 0.4  # quotients without a remainder, and one below
    num = np.where(exact, num // den * den - (rng.random(den.size) < 0.3), num).clip(0, top)
    assert _run(lib.launch_rooms, num.astype(np.int32), den.astype(np.int32)) == [0, 0]


@pytest.mark.parametrize("kind", ["screen", "grid", "half_ulp", "one_ulp", "special"])
def test_folds(lib, kind):
    rng = np.random.default_rng(len(kind))
    n = 200000
    w = rng.uniform(-1, 1, 3 * n) * 2.0 ** rng.integers(-6, 22, 3 * n)
    d = rng.uniform(-1, 1, 3 * n) * 2.0 ** rng.integers(-12, 12, 3 * n)
    if kind == "grid":
        w, d = np.round(w * 8) / 8, np.round(d * 64) / 64
    w, d = w.astype(np.float32), d.astype(np.float32)
    if kind == "half_ulp":
        d = (np.spacing(w) * (rng.integers(-9, 9, 3 * n) + 0.5)).astype(np.float32)
    elif kind == "one_ulp":  # the longest jumps: increments of a unit or two
        d = (np.spacing(w) * rng.integers(-2, 3, 3 * n)).astype(np.float32)
    elif kind == "special":
        sp = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e38, -1e38, 1e-45], np.float32)
        w[::2] = sp[rng.integers(0, 8, w[::2].size)]
        d[1::3] = sp[rng.integers(0, 8, d[1::3].size)]
    k = rng.integers(17, 16384, n).astype(np.int32)
    k[:200] = np.arange(17, 217)
    assert _run(lib.launch_folds, w, d, k) == [0, 0]
