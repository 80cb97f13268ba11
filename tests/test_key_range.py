"""How attn_row_kernel's CTAs share a row's keys (csrc/key_range.cuh, compiled for the host): the ranges follow each other without a gap, cached keys and the new
one are in one of them each, and one range alone owns the new row, also where the last ranges are empty; with -1 cached keys, a position outside the cache, all are."""
import subprocess

from tinygpt_b200 import build

MAIN = """
#include <cstdio>
#include "key_range.cuh"
int main() {
  for (int log = 0; log <= 4; ++log)
    for (int r = 0; r < 1 << log; ++r) {
      const b200::KeyRange k = b200::key_range(-1, true, r, log);
      if (k.first != 0 || k.n != 0 || k.n_cached > 0 || k.owns_new) return printf("range %d of %d without keys: %d of them\\n", r, 1 << log, k.n), 1;
    }
  for (int log = 0; log <= 4; ++log)
    for (int append = 0; append < 2; ++append)
      for (int cached = 0; cached <= 5000; cached += cached < 700 ? 1 : 37) {
        int at = 0, in_cache = 0, owners = 0;
        for (int r = 0; r < 1 << log; ++r) {
          const b200::KeyRange k = b200::key_range(cached, append, r, log);
          bool bad = k.first != at || k.n < 0;
          if (k.n > 0) in_cache += k.n_cached;
          bad = bad || (k.n > 0 && k.n_cached + (k.owns_new ? 1 : 0) != k.n);
          owners += k.owns_new;
          at += k.n;
          if (bad) return printf("range %d of %d, %d keys, append %d\\n", r, 1 << log, cached, append), 1;
        }
        if (at != cached + append || in_cache != cached || owners != append)
          return printf("%d keys, append %d, %d ranges: end %d, cached %d, owners %d\\n", cached, append, 1 << log, at, in_cache, owners), 1;
      }
  return 0;
}
"""


def test_ranges(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-I", str(build.CSRC), str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
