"""Where the CG kernel looks for its tables in shared memory (host arithmetic
shared with the kernel, cg_tables.h)."""
import os
import subprocess

import pytest

from hilbert_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cg") / "check")
    src = [os.path.join(build.CSRC, f) for f in ("cg_tables.cpp", "v2rdm_problem.cpp", "doci_problem.cpp")]
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", build.CSRC, os.path.join(HERE, "cg_tables_check.cpp"),
                           *src, "-o", exe])

    def run(*args):
        return subprocess.run([exe, *map(str, args)], capture_output=True, text=True, check=True).stdout.split("\n")
    return run


@pytest.mark.parametrize("args", [(2, 1, 1, 3), (3, 2, 1, 3 | 16), (6, 3, 3, 4), (9, 5, 4, 3), (12, 6, 6, 3),
                                  (10, 5, 5, 3, "doci")])
def test_runs_are_addressed_inside_their_own_words(check, args):
    """Every entry of a run is found inside the run's words when its index is
    added to the base as a 64-bit address, with both passes' tables side by side
    and in turn."""
    runs, wrong = (int(w.split()[0]) for w in check(*args)[0].split(", "))
    assert runs > 0 and wrong == 0


@pytest.mark.parametrize("args,per_cta,form", [((10, 5, 5, 3, "doci"), 2, "both"), ((2, 1, 1, 3), 1, "both"),
                                               ((9, 5, 4, 3), 2, "both"), ((18, 9, 9, 3), 3, "both"),
                                               ((19, 10, 9, 3), 3, "one region"), ((20, 10, 10, 3), 3, "one region"),
                                               ((22, 11, 11, 3), 1, "streamed"), ((10, 5, 5, 4), 1, "streamed")])
def test_form_of_the_kernel(check, args, per_cta, form):
    """Which problems take which form of the CG kernel on 148 SMs (227 KB of
    shared memory each): the tests of each form name their sizes by this."""
    v, got, nbytes = check(*args)[1].split(", ")
    assert (int(v.split()[0]), got) == (per_cta, form)
    assert int(nbytes.split()[0]) <= 227 * 1024 - 4096
