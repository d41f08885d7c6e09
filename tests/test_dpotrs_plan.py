"""The workspace of ooc_dpotrs_L in a caller's budget (dpotrs_plan.h), on the host: every budget from two panels, an nb x nb
inverse and 128 nb bytes on is accepted, smaller ones are refused, and what is laid out stays within it."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oocdag_gb300", "csrc")

PROGRAM = r"""
#include "dpotrs_plan.h"
#include <cstdio>
#include <initializer_list>
int main() {
  auto exchange = [](int64_t n, int r, int sweeps) { return (size_t)256 + (size_t)sweeps * n * r * 16; };
  int count = 0, bad = 0, whole = 0, split = 0;
  for (int64_t n : {1, 40, 64, 65, 300, 2000})
    for (int nb = 1; nb <= (n < 300 ? n : 300); nb++)
      for (int r : {1, 3, 8, 9, 16})
        for (int where = 0; where < 4; where++) {
          const bool l = where & 1, b = where & 2;
          const size_t least = dpotrs_plan(n, nb, r, l, b, 1, exchange).least;
          auto up = [](size_t x) { return (x + 255) / 256 * 256; };
          const size_t want = 256 + up((size_t)nb * nb * 8) + up((size_t)nb * 16 * 8) + (b ? 0 : up((size_t)n * r * 8)) +
                              (l ? 0 : 2 * up((size_t)n * nb * 8));
          bad += least != want || dpotrs_plan(n, nb, r, l, b, least - 1, exchange).ok;
          for (size_t budget : {(size_t)0, least, least + 5000, least + 200000, least + (1u << 24)}) {
            const DpotrsPlan p = dpotrs_plan(n, nb, r, l, b, budget, exchange);
            count++;
            whole += p.whole;
            split += p.group < r;
            const int64_t m = p.whole ? n : nb;
            bad += !p.ok || (budget && p.need > budget) || p.group < 1 || p.group > r || (p.whole && (!l || p.group != r));
            bad += p.inverses < exchange(m, p.group, p.whole ? 2 : 1);
            bad += p.b - p.inverses < dpotrs_inverse_bytes(m) || p.panels - p.b < (b ? 0 : (size_t)n * r * 8);
            bad += p.panel < (l ? 0 : (size_t)n * nb * 8) || p.need < p.panels + 2 * p.panel;
            bad += (p.inverses | p.b | p.panels | p.panel) % 256 != 0;
          }
        }
  printf("%d %d %d %d\n", count, bad, whole > 0, split > 0);
}
"""


def test_layouts(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-O1", "-std=c++17", "-I" + CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    count, bad, whole, split = map(int, subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split())
    assert count > 10000 and bad == 0 and whole and split


@pytest.mark.gpu
@pytest.mark.parametrize("n,nb,nrhs", [(40, 40, 16), (63, 20, 3), (130, 33, 16), (200, 63, 9), (300, 64, 16), (300, 65, 16), (400, 96, 16), (411, 137, 12)])
@pytest.mark.parametrize("where", ["device", "host"])
def test_solve_in_the_smallest_budget(handle, ooc, where, n, nb, nrhs):
    """Residual |L L^T x - b| <= 8 n 2^-53 (|L| |L^T| |x| + |b|), a multiple of substitution's componentwise bound for the factor's
    well-conditioned diagonal blocks (condition below 4, the inverses' own error)."""
    import numpy as np
    import torch

    rng = np.random.default_rng(n + nb)
    L = np.tril(rng.uniform(-0.5, 0.5, (n, n)) / np.sqrt(n)) + 2 * np.eye(n)
    B = rng.standard_normal((n, nrhs))
    least = 256 + (nb * nb * 8 + 255) // 256 * 256 + (nb * 128 + 255) // 256 * 256
    if where == "device":
        Ld, Xd = torch.from_numpy(np.ascontiguousarray(L.T)).cuda(), torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    else:
        Ld, Xd = np.asfortranarray(L), np.asfortranarray(B)
        least += (n * nrhs * 8 + 255) // 256 * 256 + 2 * ((n * nb * 8 + 255) // 256 * 256)
    with pytest.raises(ooc.OocError) as e:
        handle.dpotrs_L(Ld, n, n, nb, Xd, n, nrhs, least - 1)
    assert e.value.code == ooc.OOC_ERR_BUDGET
    handle.dpotrs_L(Ld, n, n, nb, Xd, n, nrhs, least)
    X = Xd.cpu().numpy().T if where == "device" else Xd
    bound = 8 * n * 2.0**-53 * (np.abs(L) @ (np.abs(L).T @ np.abs(X)) + np.abs(B))
    assert (np.abs(L @ (L.T @ X) - B) <= bound).all()
