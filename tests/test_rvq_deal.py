"""How tiles of vectors are dealt to pairs of blocks, and when that search is taken (csrc/fm_rvq_deal.h); no GPU needed."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "fm_rvq_deal.h"
#include <cstdio>
#include <initializer_list>
int main() {
  for (int sms : {2, 148, 400})
    for (long long rows : {1ll, 256ll, 257ll, 9472ll, 18944ll, 18945ll, 64000ll, 1000001ll})
      for (int longer : {1, 7, 32})
        for (int shorter : {0, 1, 7}) {
          if (shorter > longer) continue;
          fm::RvqDeal d;
          d.make(rows, longer, shorter, sms);
          const int tiles = static_cast<int>((rows + 255) / 256);
          int most = 0, least = 0x7fffffff;
          for (int p = 0; p < d.pairs; ++p) {
            const int n0 = d.first[0][p + 1] - d.first[0][p], n1 = d.first[1][p + 1] - d.first[1][p], load = n0 * longer + n1 * shorter;
            if (n0 < 0 || n1 < 0 || n0 + n1 < 1) return std::printf("an idle pair\n"), 1;
            most = load > most ? load : most;
            least = load < least ? load : least;
          }
          if (d.pairs < 1 || d.pairs > 80 || d.first[0][0] != 0 || d.first[1][0] != 0 || d.first[0][d.pairs] != tiles ||
              d.first[1][d.pairs] != (shorter > 0 ? tiles : 0) || most - least > longer)
            return std::printf("%d tiles, %d + %d layers, %d SMs\n", tiles, longer, shorter, sms), 1;
        }
  int rows, longer, shorter, entries;
  while (std::scanf("%d %d %d %d", &rows, &longer, &shorter, &entries) == 4) {
    fm::RvqDeal d;
    d.make(rows, longer, shorter, 148);
    std::printf("%d\n", fm::rvq_tiles_pay(d, rows, entries) ? 1 : 0);
  }
  return 0;
}
"""

# Vectors, layers (of the longer stack, of the other), entries; microseconds measured in the chain of kernels and in tiles (148 SMs).
MEASURED = [
    (2000, 1, 0, 256, 10, 23), (12000, 1, 0, 256, 14, 24), (37888, 1, 0, 256, 29, 39), (128000, 1, 0, 256, 77, 169), (12000, 2, 0, 256, 28, 34),
    (37888, 2, 0, 256, 58, 60), (6000, 8, 0, 256, 89, 98), (16000, 8, 0, 256, 129, 102), (25000, 8, 0, 256, 174, 191), (37888, 8, 0, 256, 232, 190),
    (12000, 32, 0, 256, 443, 358), (16000, 7, 1, 256, 129, 94), (64000, 7, 1, 256, 405, 407), (12000, 1, 0, 2048, 24, 34),
    (18944, 1, 0, 2048, 32, 36), (37888, 1, 0, 2048, 60, 60), (64000, 1, 0, 2048, 90, 109), (12000, 2, 0, 2048, 47, 55), (18944, 2, 0, 2048, 64, 57),
    (37888, 2, 0, 2048, 119, 103), (6000, 8, 0, 2048, 124, 175), (16000, 8, 0, 2048, 230, 182), (19200, 8, 0, 2048, 272, 336),
    (37888, 8, 0, 2048, 473, 360), (64000, 8, 0, 2048, 827, 706), (6000, 32, 0, 2048, 508, 709), (16000, 32, 0, 2048, 931, 702),
    (25000, 32, 0, 2048, 1314, 1415), (6000, 7, 1, 2048, 124, 155), (16000, 7, 1, 2048, 235, 180), (22000, 7, 1, 2048, 304, 308),
    (37888, 7, 1, 2048, 468, 394), (64000, 7, 1, 2048, 821, 683),
]


def test_tiles_are_dealt_evenly_and_taken_where_they_are_faster(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler here")
    source, program = tmp_path / "deal.cpp", tmp_path / "deal"
    source.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fast_mimi_b200", "csrc"), str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], input="\n".join(" ".join(map(str, m[:4])) for m in MEASURED), capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout
    taken = [int(line) for line in done.stdout.split()]
    assert len(taken) == len(MEASURED)
    for m, tiles in zip(MEASURED, taken):
        assert m[4 + tiles] <= 1.12 * min(m[4:]), (m, tiles)
