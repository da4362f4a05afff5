"""The chunks of a streamed host-buffer query, computed as the library does
(csrc/host_chunks.hpp): around the sizes at which its rules change and up to
the largest count, for a query first, last, both or neither in its train, they
add up to the query, none is larger than a device slot and all but the last are
whole occlusion words."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "raytracer-data-structures_gb300", "csrc")

_PROGRAM = r"""
#include <cstdio>
#include "host_chunks.hpp"
int main() {  // lines of: n begins ends -> chunks
  unsigned n, begins, ends;
  std::printf("%u\n", rq::kPipeChunk);
  while (std::scanf("%u %u %u", &n, &begins, &ends) == 3) {
    for (uint32_t c : rq::chunk_plan(n, begins != 0, ends != 0)) std::printf("%u ", c);
    std::printf("\n");
  }
}
"""

_EDGES = [1 << 19, 1 << 22, 1 << 25, 33_600_000, 40_000_000, 1 << 26, 100_000_000, 1 << 31, (1 << 32) - 1025]
_COUNTS = sorted({e + d for e in _EDGES for d in (-1, 0, 1, 33, 512, 1024)} | {1, 31, 33, 127, 128, 129, 1000})


def test_chunks_fit_their_slots(tmp_path):
    src = tmp_path / "plan.cpp"
    src.write_text(_PROGRAM)
    exe = tmp_path / "plan"
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    asked = [(n, b, e) for n in _COUNTS for b in (0, 1) for e in (0, 1)]
    r = subprocess.run([str(exe)], input="".join("%d %d %d\n" % a for a in asked), capture_output=True, text=True,
                       check=True, timeout=60)
    slot, *lines = r.stdout.splitlines()
    assert len(lines) == len(asked)
    for a, line in zip(asked, lines):
        chunks = [int(c) for c in line.split()]
        assert sum(chunks) == a[0], a
        assert min(chunks) > 0 and max(chunks) <= int(slot), (a, max(chunks))
        assert all(c % 32 == 0 for c in chunks[:-1]), a
