"""Starts of a sliced matrix's slices (csrc/slice_starts.h, host only), compiled by
the host compiler: sums past 2^31 and past 2^32 are refused, not wrapped."""

from __future__ import annotations

import shutil
import subprocess

import numpy as np
import pytest
from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "slice_starts.h"
int main(int argc, char** argv) {  // pairs: repeat size
  std::vector<int32_t> size, starts{-5};
  for (int i = 1; i + 1 < argc; i += 2) size.insert(size.end(), atoi(argv[i]), atoi(argv[i + 1]));
  printf("%lld", (long long)lapy::slice_starts(size.data(), (int)size.size(), &starts));
  for (int32_t s : starts) printf(" %d", s);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("slice_starts")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", f"-I{ROOT / 'lapy_gb300' / 'csrc'}", str(d / "main.cpp"),
                    "-o", str(d / "main")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("runs", [[], [(3, 0)], [(2, 64), (1, 0), (3, 192)], [(1, 2**31 - 1)], [(1023, 2**21), (1, 64)],
                                  [(1, 2**31 - 64), (1, 64)], [(2**10, 2**21)], [(2**11, 2**21), (1, 128)],
                                  [(2**12, 2**21), (5, 64)]])
def test_sums(program, runs):
    out = subprocess.run([program, *(str(x) for r in runs for x in r)], check=True, capture_output=True, text=True)
    total, *starts = (int(x) for x in out.stdout.split())
    size = np.concatenate([np.zeros(0, np.int64), *(np.full(r, s, np.int64) for r, s in runs)])
    if size.sum() >= 2**31:
        assert total == -1 and starts == [-5]  # untouched
    else:
        assert total == size.sum() and starts == [0, *np.cumsum(size).tolist()]


def test_both_matrix_copies_use_it():
    for name in ("pcg.cu", "pcg_cluster.cu"):
        text = (ROOT / "lapy_gb300" / "csrc" / name).read_text()
        assert text.count("slice_starts(") == 1
