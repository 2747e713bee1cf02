"""Work on several streams is joined whatever fails (csrc/fork_join.h, host only),
compiled by the host compiler with fakes of the launch and of the wait."""

from __future__ import annotations

import shutil
import subprocess

import pytest
from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "fork_join.h"
int main(int argc, char** argv) {
  const int n = atoi(argv[1]), bad_begin = atoi(argv[2]), bad_join = atoi(argv[3]);
  const int status = lapy::fork_join(
      n, [&](int i) { printf("b%d ", i); return i == bad_begin ? -2 : 0; },
      [&](int i) { printf("j%d ", i); return i == bad_join ? -9 : 0; });
  printf("%d\n", status);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("fork_join")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", f"-I{ROOT / 'lapy_gb300' / 'csrc'}", str(d / "main.cpp"),
                    "-o", str(d / "main")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("n", [0, 1, 2, 5])
@pytest.mark.parametrize("bad_begin", [-1, 0, 1, 4])
@pytest.mark.parametrize("bad_join", [-1, 0, 3])
def test_every_piece_begun_is_joined(program, n, bad_begin, bad_join):
    out = subprocess.run([program, str(n), str(bad_begin), str(bad_join)], check=True, capture_output=True, text=True)
    *calls, status = out.stdout.split()
    begun = n if not 0 <= bad_begin < n else bad_begin + 1
    assert calls == [f"b{i}" for i in range(begun)] + [f"j{i}" for i in range(begun)]
    want = -2 if 0 <= bad_begin < n else -9 if 0 <= bad_join < begun else 0
    assert int(status) == want


def test_the_on_chip_solver_forks_through_it():
    """Each launch of its classes and each wait of the caller's stream."""
    text = (ROOT / "lapy_gb300" / "csrc" / "pcg_cluster.cu").read_text()
    body = text[text.index("int cluster_solve("):]
    assert body.count("cudaLaunchKernelEx") == 1 and body.count("fork_join(") == 1
    assert body.index("fork_join(") > body.index("auto begin") > 0
