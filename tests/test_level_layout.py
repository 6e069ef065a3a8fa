"""The layout of the structures that C callers pass: arrays of them are walked
with the library's stride, so a published structure never grows."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

from glide_b200 import _native as N

INCLUDE = Path(__file__).resolve().parent.parent / "include"
# bytes on x86-64
SIZES = {"GlideLevelArgs": 144, "GlideLevel": 328, "GlideSolverConfig": 136}


def test_published_sizes(tmp_path):
    cc = shutil.which("g++")
    if not cc:
        pytest.skip("no C++ compiler")
    src = tmp_path / "s.cpp"
    src.write_text('#include "glide_b200.h"\n#include <cstdio>\nint main() { std::printf("%zu %zu %zu\\n", '
                   'sizeof(GlideLevelArgs), sizeof(GlideLevel), sizeof(GlideSolverConfig)); }\n')
    subprocess.run([cc, "-I", str(INCLUDE), str(src), "-o", str(tmp_path / "s")], check=True)
    out = subprocess.run([str(tmp_path / "s")], check=True, capture_output=True, text=True).stdout.split()
    assert [int(x) for x in out] == list(SIZES.values())


def test_bindings_have_the_same_sizes():
    assert [C.sizeof(t) for t in (N.LevelArgs, N.Level, N.SolverConfig)] == list(SIZES.values())
