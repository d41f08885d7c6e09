"""The FP32 trailing update's choice between digit planes and the FP32 pipe (syrk32_way.h), on the host with a buffer
whose growth can be made to fail: a panel's later block-column ranges follow the choice made when it was prepared, so planes
that found no room are never read."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oocdag_gb300", "csrc")

PROGRAM = r"""
#include "syrk32_way.h"
#include <cstdio>
#include <initializer_list>
struct Buf {
  size_t limit, bytes = 0;
  int ensure(size_t b) {  // like a device buffer: a failed growth leaves none
    if (b <= bytes) return 0;
    bytes = 0;
    if (b > limit) return -5;
    bytes = b;
    return 0;
  }
};
int main() {
  const size_t digits = 4096, copy = 2048;
  auto planes_of = [](int64_t rows, int k) { return (size_t)rows * k * 8; };
  auto chunked = [](int64_t rows, int k) { return (size_t)((rows + 127) / 128) * 128 * (size_t)(k < 512 ? k : 512) * 8; };
  for (int64_t n : {1, 100, 511, 512, 513, 1000, 6001})
    for (int nb : {64, 256, 384, 512})
      for (int w = nb % 256 ? 64 : 128; w <= nb; w *= 2)
        printf("m %lld %d %d: %zu\n", (long long)n, nb, w, syrk32_largest(n, nb, w, chunked));
  for (int64_t n : {100, 1000, 6000})
    for (int nb : {64, 100, 512})
      for (size_t budget = 0; budget <= (size_t)12 * n * 8 * nb; budget += (size_t)n * nb) {
        bool planes = false;
        const int64_t W = spotrf_ooc_width(n, nb, budget, planes_of, 512, &planes);
        printf("w %lld %d %zu: %lld %d\n", (long long)n, nb, budget, (long long)W, (int)planes);
      }
  for (size_t limit : {(size_t)0, copy, digits})
    for (int serve = 0; serve < 2; serve++)
      for (int aligned = 0; aligned < 2; aligned++) {
        Buf b{limit};
        Syrk32Way way = Syrk32Way::kNone;
        const int rc = syrk32_choose(b, serve, digits, aligned, copy, &way);
        printf("c %zu %d %d: %d %d %zu\n", limit, serve, aligned, rc, (int)way, b.bytes);
      }
}
"""


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("way")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I" + CSRC, str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    out = subprocess.run([str(d / "t")], check=True, capture_output=True, text=True).stdout
    rows = [line.split(": ") for line in out.strip().splitlines()]
    return {(k[0], *map(int, k[2:].split())): tuple(map(int, v.split())) for k, v in rows}


NONE, DIRECT, COPIED, DIGITS = range(4)


def test_every_choice(table):
    choices = {k[1:]: v for k, v in table.items() if k[0] == "c"}
    assert len(choices) == 12
    for (limit, serve, aligned), (rc, way, held) in choices.items():
        if serve and limit >= 4096:
            want = (0, DIGITS, 4096)
        elif aligned:
            want = (0, DIRECT, 0)
        elif limit >= 2048:
            want = (0, COPIED, 2048)
        else:
            want = (-5, NONE, 0)
        assert (rc, way, held) == want, (limit, serve, aligned)


def test_out_of_core_width_and_planes_stay_within_the_budget(table):
    rows = {k[1:]: v for k, v in table.items() if k[0] == "w"}
    assert len(rows) > 500 and {p for _, p in rows.values()} == {0, 1}
    for (n, nb, budget), (W, planes) in rows.items():
        widest = budget // (12 * n) // nb * nb
        assert W % nb == 0 and (W == 0) == (widest < nb)  # what was accepted stays accepted
        if W == 0:
            continue
        fits = [w for w in range(nb, widest + 1, nb) if 4 * w >= 3 * widest and 12 * n * w + 8 * n * min(w, 512) <= budget]
        assert (W, planes) == ((max(fits), 1) if fits else (widest, 0)), (n, nb, budget)


def test_the_first_reservation_holds_every_update(table):
    """Panels of w columns inside tiles of nb: the rest of a tile takes each panel, everything right of it the whole tile."""
    rows = {k[1:]: v[0] for k, v in table.items() if k[0] == "m"}
    assert len(rows) > 40
    for (n, nb, w), reserved in rows.items():
        most = 0
        for j in range(0, n, w):
            end, tile = min(j + w, n), min(j // nb * nb + nb, n)
            if end < n:
                k = end - j if end < tile else tile - j // nb * nb
                most = max(most, -(-(n - end) // 128) * 128 * min(k, 512) * 8)
        assert most <= reserved, (n, nb, w)
        assert reserved <= -(-n // 128) * 128 * min(nb, 512) * 8
