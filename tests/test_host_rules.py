"""Host-compiled checks of rules the kernels share with the host: small programs around the headers of csrc/,
built with nvcc and run on the CPU."""
import os
import subprocess

from svoo_b200 import build

MAP_READS = r"""
#include <cstdio>
#include "map_common.cuh"
// Every read, at every alignment of maps of 1 to 5 rows: it lies inside the map, and the bytes are the map's.
struct Recorder {
  const uint8_t *lo, *hi;
  mutable bool outside = false;
  uint32_t word(const uint8_t* p) const {
    outside |= p < lo || p + 4 > hi || reinterpret_cast<uintptr_t>(p) % 4;
    return p[0] | p[1] << 8 | p[2] << 16 | (uint32_t)p[3] << 24;
  }
  uint32_t byte(const uint8_t* p) const {
    outside |= p < lo || p >= hi;
    return *p;
  }
};
int main() {
  alignas(8) static uint8_t mem[4096];
  const int rows_of[] = {1, 2, 5}, cols_of[] = {1, 2, 3, 4, 5, 31, 32, 33, 63, 65, 97, 500};
  for (int rows : rows_of)
    for (int KC : cols_of)
      for (int place = 64; place < 68; ++place) {
        const int total = rows * KC;
        uint8_t* map = mem + place;
        for (int i = 0; i < total; ++i) map[i] = (uint8_t)(i * 37 % 3);
        const Recorder load{map, map + total};
        for (int r = 0; r < rows; ++r)
          for (int lane = 0; lane < 32; ++lane) {
            const int j0 = lane * 32, left = KC - j0, bytes = left < 0 ? 0 : (left > 32 ? 32 : left);
            uint32_t w[9];
            const int skew = svoo::map_words(w, map + r * KC + j0, bytes, map, map + total, load);
            for (int b = 0; b < bytes; ++b)
              if ((w[(b + skew) / 4] >> (8 * ((b + skew) % 4)) & 0xFF) != map[r * KC + j0 + b]) return printf("wrong byte\n"), 1;
          }
        if (load.outside) return printf("read outside: %d x %d at %d\n", rows, KC, place), 1;
      }
  puts("ok");
  return 0;
}
"""


SORT_RULE = r"""
#include <cstdio>
#include "common.cuh"
// The sort takes the largest cluster that the size asks for and the device can place.
int main() {
  const long sizes[][3] = {{1, 1, 1}, {2, 4096, 32}, {12, 32760, 500}, {40, 75600, 500}, {3, 40003, 1024}, {64, 75600, 100}, {300, 75600, 100}};
  const int want[] = {1, 8, 16, 8, 16, 8, 1};
  for (int i = 0; i < 7; ++i)
    for (int limit = 1; limit <= 16; limit *= 2) {
      const int got = svoo::sort_cluster_ctas(sizes[i][0], sizes[i][1], sizes[i][2], 148, [&](int ctas) { return ctas <= limit; });
      if (got != (want[i] < limit ? want[i] : limit)) return printf("%d %d: %d\n", i, limit, got), 1;
    }
  puts("ok");
  return 0;
}
"""


def _run(tmp_path, source):
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(source)
    res = subprocess.run([build._nvcc(), "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", build.CSRC,
                          str(src), "-o", str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout)


def test_map_words_stay_inside_the_map(tmp_path):
    _run(tmp_path, MAP_READS)


def test_sort_takes_a_cluster_that_fits(tmp_path):
    _run(tmp_path, SORT_RULE)
