"""The work split of the tensor-core kernels (WorkLine in csrc/fsk_tc.cuh), host
side: every data tile of every query block belongs to one segment of one CTA,
segment numbers are unique and those the reductions read, and sizes past 2^31
tiles per CTA stay in range."""
import shutil
import subprocess

from conftest import PKG

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "fsk_tc.cuh"
using namespace fsk;
using tc::WorkLine;

static WorkLine line(int64_t q_blocks, int64_t n_tiles, int sms) {
  WorkLine w;
  w.n_tiles = n_tiles;
  w.grid = (int)(q_blocks * n_tiles < sms ? q_blocks * n_tiles : sms);
  w.whole = (int)(q_blocks / w.grid);
  w.rest = (int)(q_blocks % w.grid);
  const int64_t share = w.rest * n_tiles < w.grid ? w.rest * n_tiles : w.grid;
  w.line_grid = (int)(share > 1 ? share : 1);
  return w;
}

#define CHECK(c) if (!(c)) { printf("%s at %lld blocks, %lld tiles, %d SMs\n", #c, (long long)qb, (long long)nt, sms); exit(1); }

static void check(int64_t qb, int64_t nt, int sms, bool every_tile) {
  const WorkLine w = line(qb, nt, sms);
  std::vector<char> seen(every_tile ? qb * nt : 0), number(every_tile ? w.segment_bound() : 0);
  int64_t total = 0;
  for (int b = 0; b < w.grid; ++b) {
    for (int k = 0;; ++k) {
      const tc::Segment g = tc::segment_at(w, b, k);
      if (g.count == 0) break;
      CHECK(g.qb >= 0 && g.qb < qb && g.t0 >= 0 && g.count > 0 && (int64_t)g.t0 + g.count <= nt);
      const int64_t id = w.segment_id(g.qb, b);
      CHECK(id >= 0 && id < w.segment_bound());
      int n;
      const int64_t first = w.segments_of(g.qb, n);
      CHECK(id >= first && id < first + n);
      total += g.count;
      if (!every_tile) continue;
      CHECK(!number[id]);
      number[id] = 1;
      for (int t = 0; t < g.count; ++t) {
        CHECK(!seen[g.qb * nt + g.t0 + t]);
        seen[g.qb * nt + g.t0 + t] = 1;
      }
    }
  }
  CHECK(total == qb * nt);
  if (!every_tile) return;
  int64_t rows = 0, used = 0;
  for (int64_t q = 0; q < qb; ++q) {
    int n;
    w.segments_of(q, n);
    rows += n;
  }
  for (char c : number) used += c;
  CHECK(rows == used);
}

int main() {
  for (int sms : {1, 7, 148, 152})
    for (int64_t qb : {1, 2, 3, 8, 40, 147, 151, 152, 153, 300, 305})
      for (int64_t nt : {1, 2, 3, 5, 64, 157, 400}) check(qb, nt, sms, true);
  // 1e8 and 2e8 points at as many queries (256 queries a block, 64 or 128 points
  // a tile), a short set of data at very many queries and the reverse
  for (int64_t n : {100000000ll, 200000000ll, 1073741824ll})
    for (int64_t tile : {64, 128}) check((n + 255) / 256, (n + tile - 1) / tile, 152, false);
  check(4000000, 1000000, 152, false);
  check(1, 2000000000ll, 152, false);
  check(8000000, 1, 152, false);
  puts("ok");
}
"""


def test_work_line(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "line.cu", tmp_path / "line"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-O1", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", str(PKG / "csrc"),
                    "-I", str(PKG.parent / "include"), "-o", str(exe), str(src)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr
