"""The adjoint's cell and face reverses at spacings dx != dy, both other than 1, in the form with divisions and in
the one with reciprocals (powers of two), against central differences on the CPU; and that the reverse checked
there is made of the functions the kernels run."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "microsim_b200", "csrc")
TAGS = ("quotient", "quotient2", "product", "product4")
CHECKS = ("dphi_obstacle", "dphi_well", "dphi_projected", "flux_x", "flux_y", "current_obstacle_x", "current_obstacle_y",
          "current_well_x", "current_well_y", "mu")


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("adj") / "adj_spacing_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", CSRC, "-o", exe, os.path.join(HERE, "adj_spacing_check.cpp")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {line.split()[0]: float(line.split()[1]) for line in out.splitlines()}


@pytest.mark.parametrize("check", CHECKS)
@pytest.mark.parametrize("tag", TAGS)
def test_reverse_matches_differences(results, tag, check):
    assert results[f"{tag}_{check}"] < 1e-5  # rounding of the differences: 1e-16 / 1e-6, and h^2 terms


@pytest.mark.parametrize("tag", TAGS)
def test_the_projection_is_reached(results, tag):
    assert results[tag + "_cut"] > 50


def test_the_checked_reverses_are_the_kernels():
    """Every function of the header is reached from a kernel; dphi_rev and fface_rev, which run a cell's lanes or a
    face's two sides one after the other, are for these checks and call nothing else."""
    with open(os.path.join(CSRC, "gp_adjoint_cell.cuh")) as f:
        head = re.sub(r"//[^\n]*", "", f.read())
    with open(os.path.join(CSRC, "gp_adjoint.cu")) as f:
        reached = set(re.findall(r"\b(\w+)\s*(?:<[\w, ]*>)?\(", f.read()))
    starts = [(m.start(), m.group(1)) for m in re.finditer(r"\nGP_HD [\w<>]+ (\w+)\(", head)]
    calls = {}
    for (at, name), end in zip(starts, [s[0] for s in starts[1:]] + [len(head)]):
        calls[name] = set(re.findall(r"\b(\w+)\(", head[at + len(name) + 7:end])) - {name}
    known = set(calls)
    todo = list(reached & known)
    reached = set(todo)
    while todo:
        for n in calls[todo.pop()] & known - reached:
            reached.add(n)
            todo.append(n)
    assert known - reached == {"dphi_rev", "fface_rev"}
    for n in ("dphi_rev", "fface_rev"):
        assert calls[n] & known <= reached
