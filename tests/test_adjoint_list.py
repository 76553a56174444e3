"""The adjoint's list kernels visit every item of a list whose faces, or whose last stride, pass 32 bits (a
grid of 23,170 x 23,170 cells with phi varying in every cell): the walk they share, run on the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
TOP = 2**31 - 1
CASES = {"empty": (0, 4, 0, 75776), "one": (1, 4, 3, 75776), "faces_below": (2**29 - 1, 4, 5, 75776),
         "faces_at": (2**29, 4, 5, 75776), "faces_top": (TOP, 4, 75775, 75776), "cells_top": (TOP, 1, 9468, 9472)}


@pytest.fixture(scope="module")
def walks(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("walk") / "adj_list_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", os.path.join(os.path.dirname(HERE), "microsim_b200", "csrc"),
                    "-o", exe, os.path.join(HERE, "adj_list_check.cpp")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {f[0]: (int(f[1]), int(f[2])) for f in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("name", CASES)
def test_every_item_is_visited(walks, name):
    cells, per, first, step = CASES[name]
    items = range(first, cells * per, step)
    assert walks[name] == (len(items), items[-1] if items else -1)
