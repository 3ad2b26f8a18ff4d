"""Walks over slots near the largest one a graph can have (2m = 2^32 - 2): every slot of the run is
visited once and the walk ends.  The device header is compiled for the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "pb_walk.cuh"

static std::vector<int> seen;
static uint32_t beg, len;
static long calls;

static void visit(uint32_t slot, bool valid) {
  if (++calls > 100000) { puts("does not end"); exit(1); }
  if (!valid) return;
  if (slot - beg >= len) { printf("slot %u outside\n", slot); exit(1); }
  ++seen[slot - beg];
}

template <class Walk>
static void check(const char* what, Walk&& walk) {
  seen.assign(len, 0);
  calls = 0;
  walk();
  for (uint32_t t = 0; t < len; ++t)
    if (seen[t] != 1) { printf("%s: slot %u of %u + %u seen %d times\n", what, beg + t, beg, len, seen[t]); exit(1); }
}

template <int kStride>
static void strided() {
  check("turns", [&] {
    for (uint32_t first = 0; first < kStride; ++first)
      pb::walk_turns<kStride>(beg, len, first, [](uint32_t slot, int32_t left) {
        for (int r = 0; r < 4; ++r) visit(slot + r * kStride, left > r * kStride);
      });
  });
}

int main() {
  const uint32_t end = 0xFFFFFFFEu;  // one behind the last slot
  for (uint32_t n : {1u, 31u, 32u, 33u, 500u, 2047u, 2048u, 2049u, 6000u})
    for (uint32_t back : {0u, 1u, 31u, 300u}) {
      len = n;
      for (uint32_t b : {end - back - n, 7u}) {
        beg = b;
        strided<32>();
        strided<128>();
        strided<512>();
        for (uint32_t group : {32u, 128u, 512u})
          check("groups", [&] {
            for (uint32_t at = 0; at < group; ++at) pb::walk_groups(beg, len, group, at, visit);
          });
      }
    }
  puts("ok");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_walks_end_at_the_last_slots(tmp_path):
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "parbutterfly_b200", "csrc"), "-o", str(exe),
                    str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert (r.returncode, r.stdout.strip()) == (0, "ok"), r.stdout
