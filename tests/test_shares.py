"""How the steps of a persistent kernel are dealt out to its blocks (csrc/fm_shares.h); no GPU needed."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "fm_shares.h"
#include <initializer_list>
#include <cstdio>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s (sequences %d of %d tiles, %d blocks)\n", __LINE__, #x, seqs, tiles, blocks); return 1; } } while (0)
int main() {
  for (int blocks : {1, 2, 7, 132, 148})
    for (int seqs = 8; seqs <= 400; seqs += 8)
      for (int tiles : {3, 4, 5, 8, 12, 20, 79}) {
        const fm::Shares s(seqs, tiles, blocks);
        const int n = seqs * tiles, used = s.used(), most = (n + blocks - 1) / blocks;
        CHECK(used >= 1 && used <= blocks && used <= n);
        int at = 0, crossing = 0, inside = 0;
        for (int b = 0; b < used; ++b) {
          int seq, tile, steps;
          s.share(b, &seq, &tile, &steps);
          CHECK(tile >= 0 && tile < tiles && seq * tiles + tile == at && steps >= 1 && steps <= most);
          at += steps;
          crossing += tile + steps > tiles;
          inside += tile != 0;
        }
        CHECK(at == n);
        // whole sequences, or parts of one, wherever that takes no block more steps than the fewest
        if (most % tiles == 0) CHECK(inside == 0);
        if (seqs * ((tiles + most - 1) / most) <= blocks) CHECK(crossing == 0);
      }
  const int seqs = 0x7ffffff8 / 3 / 8 * 8, tiles = 3, blocks = 148;      // as many steps as an int can count
  int seq, tile, steps;
  const fm::Shares most(seqs, tiles, blocks);
  most.share(most.used() - 1, &seq, &tile, &steps);
  CHECK(seq * 3 + tile + steps == seqs * 3 && steps > 0 && most.used() <= blocks);
  std::puts("ok");
  return 0;
}
"""


def test_shares_cover_every_step_and_keep_to_sequences(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler here")
    source, program = tmp_path / "shares.cpp", tmp_path / "shares"
    source.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fast_mimi_b200", "csrc"), str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0 and done.stdout.strip() == "ok", done.stdout


DEALT = r"""
#include "fm_shares.h"
#include <cstdio>
int main() {
  int clips;
  while (std::scanf("%d", &clips) == 1) std::printf("%d\n", fm::dealt_heads_pay(fm::Shares(clips, 8, 74), clips, 74) ? 1 : 0);
  return 0;
}
"""

# Clips of 226 to 250 frames; microseconds a call on new inputs measured with whole clips in turn and with heads dealt (74 pairs of blocks).
CLIPS = [(1, 42.6, 19.2), (64, 44.2, 43.0), (75, 75.9, 51.0), (100, 80.0, 63.5), (129, 80.6, 78.9), (138, 84.1, 85.1), (149, 108.6, 86.7), (203, 119.7, 120.5),
         (209, 126.6, 129.7), (268, 157.5, 156.5), (277, 162.0, 163.5), (286, 163.9, 169.1), (340, 200.6, 201.6), (350, 205.9, 209.4), (408, 236.9, 239.5),
         (468, 277.0, 274.2), (490, 285.1, 289.3), (500, 288.1, 297.7)]


def test_heads_are_dealt_where_that_is_faster(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler here")
    source, program = tmp_path / "dealt.cpp", tmp_path / "dealt"
    source.write_text(DEALT)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fast_mimi_b200", "csrc"), str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], input="\n".join(str(c[0]) for c in CLIPS) + "\n74 148 512", capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout
    dealt = [int(line) for line in done.stdout.split()]
    assert dealt[len(CLIPS):] == [0, 0, 0]              # whole clips come out even
    for clip, taken in zip(CLIPS, dealt):
        assert clip[1 + taken] <= 1.002 * min(clip[1:]), clip
