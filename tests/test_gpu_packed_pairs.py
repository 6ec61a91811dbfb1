"""The packed float functions that the mixed FV 2D and Hermite 2D kernels run give, in both halves, the bits
of the scalar functions behind the float pointwise entry points (which test_gpu_pointwise.py checks):
smooth, noisy, jumping, constant, tiny (subnormal) and huge data, NaN and infinities, the halves of a pair
different.  Exact: the same operations, rounded the same."""
from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent
WHAT = ["teno5", "teno5i", "routed", "routed_minus", "linear", "weno5js", "weno5z", "weno5n", "teno5n", "teno5a", "gl3",
        "left_x", "left_y", "right_x", "right_y", "hllc_x", "hllc_y", "rusanov_x", "rusanov_y", "hteno", "teno5_cross"]
HERMITE = ["gl3", "left_x", "left_y", "right_x", "right_y", "hteno", "teno5_cross"]
FV = [w for w in WHAT if w not in ("hteno", "teno5_cross")]


def compile_unit(tmp: Path, unit: int) -> Path:
    from hteno import build as b

    out = tmp / f"packed{unit}.so"
    cmd = [str(b._cuda_home() / "bin" / "nvcc"), *b.ARCH, *b.NVCC_FLAGS, f"-DUNIT={unit}", "-I", str(REPO / "include"),
           *(["--fmad=false"] if unit == 0 else []), "-shared", "-o", str(out),
           str(REPO / "tests" / "cuda" / "packed_pairs.cu"), str(b.CSRC / "device_consts.cpp")]
    done = subprocess.run(cmd, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    return out


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("packed")
    libs = []
    for unit in (0, 1):
        lib = ctypes.CDLL(str(compile_unit(tmp, unit)))
        lib.packed_mismatches.argtypes = [ctypes.c_int, ctypes.c_long, ctypes.c_ulonglong]
        lib.packed_mismatches.restype = ctypes.c_long
        libs.append(lib)
    return libs


def test_compiles(tmp_path):
    for unit in (0, 1):
        assert compile_unit(tmp_path, unit).exists()


@pytest.mark.gpu
@pytest.mark.parametrize("unit,what", [(0, w) for w in FV] + [(1, w) for w in HERMITE])
def test_packed_equals_scalar(hteno_lib, cuda, units, unit, what):
    for seed, n in ((1, 2), (2, 130), (3, 1 << 22), (4, 1 << 22)):
        assert units[unit].packed_mismatches(WHAT.index(what), n, seed) == 0
