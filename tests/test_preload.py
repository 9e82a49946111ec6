"""A row-stage kernel whose shared memory the driver refuses is an error of the
context's creation, not of whatever launch comes across it later."""

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    out = tmp_path_factory.mktemp("preload") / "libpreload.so"
    csrc = ROOT / "pdf-raster_b200" / "csrc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-std=c++17",
                    "-shared", "-Xcompiler", "-fPIC", "-I", str(ROOT / "include"), "-o", str(out),
                    str(ROOT / "tests" / "preload_shim.cu"), str(csrc / "rrb_stroke.cpp")], check=True, cwd=str(ROOT))
    return C.CDLL(str(out))


@pytest.mark.parametrize("fail", [0, 1, 3, 5])
def test_a_refused_setting_is_reported(shim, fail):
    calls = C.c_int()
    assert (shim.pl_preload(fail, C.byref(calls)) != 0) == (fail != 0)
    assert calls.value == 5  # every row-stage shape is asked for
