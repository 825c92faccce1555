"""The layout of a centroid-scoring call (csrc/mvr_plan.hpp), compiled for the host:
the memory of its lists over token counts, probe counts and centroid counts."""
import os
import subprocess

from helpers import ROOT

SOURCE = r"""
#include <cstdio>
#include "mvr_plan.hpp"
using namespace mvr;
int main() {
  const int n_sm = 148;
  for (uint32_t n_cent : {1u, 1000u, 8192u, 65536u, 262144u})
    for (uint32_t nprobe : {1u, 2u, 4u, 7u, 8u, 9u, 16u, 17u, 32u}) {
      size_t most = 0;
      uint32_t at = 0, bad = 0;
      for (uint64_t n = 1; n < (1u << 21); n = n < 512 ? n + 1 : n + n / 97 + 1)
        for (uint32_t part = 1; part <= 4 && (part == 1 || part * 4096 <= n); part++) {
          const uint32_t chunk = score_chunk((uint32_t)n, n_cent, nprobe, n_sm, part);
          if (chunk == 0) { bad++; continue; }
          for (uint32_t t : {(uint32_t)(n < chunk ? n : chunk), (uint32_t)(n % chunk)}) {
            if (t == 0) continue;
            const ProbePlan p = probe_plan(t, n_cent, nprobe, n_sm);
            const size_t b = p.n_ent * 16 + p.n_gid * 4 + p.n_cnt * 4;
            if (b > most) { most = b; at = t; }
            const uint32_t n_tiles = (n_cent + 127) / 128;
            if (p.splits * p.tiles_per_split < n_tiles || (p.splits - 1) * p.tiles_per_split >= n_tiles ||
                p.k < nprobe || (t + 255) / 256 > 65535)
              bad++;
          }
        }
      std::printf("%u %u %zu %u %u\n", n_cent, nprobe, most, at, bad);
    }
}
"""


def test_lists_stay_within_their_limit(tmp_path):
    src = tmp_path / "plan.cpp"
    src.write_text(SOURCE)
    csrc = os.path.join(ROOT, "multi-vector-retrieval-gpu_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", csrc, "-o", tmp_path / "plan", src], check=True)
    out = subprocess.run([tmp_path / "plan"], check=True, capture_output=True, text=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) == 45
    for n_cent, nprobe, most, at, bad in rows:
        assert bad == 0, (n_cent, nprobe)
        assert most <= 800_000_000, (n_cent, nprobe, at)
