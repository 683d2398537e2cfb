"""Host logic of segment plans, no device: window records whose windows are
wider than the longest short vector (a Scan's: windows of 47/64 of a tile,
vectors of up to a quarter), through the library's own builder."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
namespace scl {
void segplan_window_records(const uint64_t* off, uint64_t n_seg, uint64_t short_max, uint64_t window,
                            std::vector<uint64_t>* rec);
}
#define CHECK(c) do { if (!(c)) { std::printf("case %d: %s\n", t, #c); return 1; } } while (0)
int main() {
  std::mt19937_64 rng(7);
  const uint64_t tiles[] = {64, 1024, 8192, 32768};
  for (int t = 0; t < 400; ++t) {
    const uint64_t tile = tiles[t % 4], short_max = tile / 4, window = tile * 47 / 64;
    const uint64_t most[] = {2, short_max / 8 + 1, short_max + 2, 3 * short_max};
    std::vector<uint64_t> off{rng() % 3 ? 0 : rng() % tile};
    for (int s = 0; s < 700; ++s) {
      const uint64_t edge[] = {0, short_max, short_max + 1, window, 1};
      off.push_back(off.back() + (rng() % 8 ? rng() % most[(t / 4) % 4] : edge[rng() % 5]));
    }
    const uint64_t n = off.size() - 1;
    std::vector<uint64_t> rec;
    scl::segplan_window_records(off.data(), n, short_max, window, &rec);
    std::vector<int> owners(n, 0);
    uint64_t prev = 0;
    for (size_t r = 0; r < rec.size(); r += 4) {
      const uint64_t first = rec[r], end = rec[r + 1];
      CHECK(prev <= first && first < end && end <= n);
      prev = end;
      CHECK(rec[r + 2] == off[first] && rec[r + 3] == off[end] - off[first]);
      CHECK(rec[r + 3] <= tile);  // fits in a staged tile
      for (uint64_t s = first; s < end; ++s) {
        ++owners[s];
        CHECK(off[s] / window == off[first] / window);   // starts in one window
        CHECK(s + 1 == end || off[s + 1] <= (off[first] / window + 1) * window);
      }
      // no record could have gone on
      if (end < n && off[end + 1] - off[end] <= short_max) CHECK(off[end] / window != off[first] / window);
    }
    for (uint64_t s = 0; s < n; ++s) CHECK(owners[s] == (off[s + 1] - off[s] <= short_max ? 1 : 0));
  }
  return 0;
}
"""


def test_scan_window_records(built, tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    (tmp_path / "t.cpp").write_text(SOURCE)
    lib = ROOT / "skelcl_gb300"
    subprocess.run(["g++", "-std=c++17", "-O1", "t.cpp", "-o", "t", f"{lib}/libskelcl_cuda.so", f"-Wl,-rpath,{lib}"],
                   cwd=tmp_path, check=True)
    r = subprocess.run(["./t"], cwd=tmp_path, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
