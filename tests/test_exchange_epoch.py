"""The tags of the triangular solves' exchange buffer (exchange_epoch.h), on the host: a launch whose wait ran out leaves the
buffer's error word raised, which would end every later launch at its first ticket, so the next solve with that factor
has to start on a zeroed buffer; so has the one after every tag has been used."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oocdag_gb300", "csrc")

PROGRAM = r"""
#include "exchange_epoch.h"
#include <cstdio>
int main() {
  ExchangeEpoch e;
  auto show = [&](const char* what) {
    bool clear = false;
    const unsigned tag = e.next(&clear);
    printf("%s %u %d\n", what, tag, (int)clear);
  };
  show("new");
  show("second");
  show("third");
  e.restart();
  show("failed");
  show("after");
  e = ExchangeEpoch(0xfffffffeu);
  show("last");
  show("wrapped");
}
"""


def test_tags(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split("\n")
    assert out[:7] == ["new 1 1", "second 2 0", "third 3 0", "failed 1 1", "after 2 0", "last 4294967295 0", "wrapped 1 1"]


def test_every_solve_of_a_factor_ends_in_its_status():
    """Whatever reads a factor's error word hands it, and any failure, to the factor."""
    text = open(os.path.join(CSRC, "mixed.cu")).read()
    reads = len(re.findall(r"queue_solve_error\(F->xch", text))
    assert reads and reads == len(re.findall(r"= factor_solve_status\(F|return factor_solve_status\(F", text))
