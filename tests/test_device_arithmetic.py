"""The kernels' own small functions (j_presto_b200/csrc/jp_common.cuh), compiled for the host and run
there: the reciprocal-square-root step of the FP64 pair kernel, the bit orders of the pair
records' masks and the 16-bit type words.
"""
import os
import shutil
import subprocess

import pytest

from j_presto_b200 import build

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "jp_common.cuh"
using namespace jp;

// largest error of rsqrt_step in 2^-53, starts off by up to 2^-20 either way
static double step_error(std::mt19937_64& rng) {
  std::uniform_real_distribution<double> u(-1.0, 1.0), m(1.0, 4.0);
  double worst = 0.0;
  for (int i = 0; i < 400000; ++i) {
    const double x = std::ldexp(m(rng), 2 * (int)(rng() % 40) - 40);
    const long double r = 1.0L / sqrtl((long double)x);
    const double off = i % 4 == 0 ? (u(rng) < 0 ? -1.0 : 1.0) : u(rng);
    const double y = (double)(r * (1.0L + std::ldexp(1.0L, -20) * off));
    const long double err = fabsl((long double)rsqrt_step(x, y) / r - 1.0L);
    worst = std::fmax(worst, (double)(err * 0x1p53L));
  }
  return worst;
}

// every listed (i atom, entry) pair of a record is met once and no other: lane l of eight, i atoms l
// and l + 8, meets at step k of group g entry 8 g + ((l + k) & 7)
static int order_faults(std::mt19937_64& rng) {
  int bad = 0;
  for (int t = 0; t < 2000; ++t) {
    unsigned row[16], met[16] = {0};
    for (int r = 0; r < 16; ++r) row[r] = t == 0 ? 0xffffffffu : t == 1 ? 1u << (r + 8) : (unsigned)rng();
    for (int r = 0; r < 16; ++r) {
      const int l = r & 7;
      const unsigned word = record_row(row[r], r), m = step_mask(word, r);
      for (int g = 0; g < 4; ++g)
        for (int k = 0; k < 8; ++k)
          if ((m >> (8 * g + k)) & 1u) met[r] |= 1u << (8 * g + ((l + k) & 7));
      bad += __builtin_popcount(m) != __builtin_popcount(row[r]) || met[r] != row[r];
      // one i atom a lane: bit k is entry (r + k) & 15, bit 16 + k is 16 + ((r + k) & 15)
      for (int k = 0; k < 16; ++k) {
        const int e = (r + k) & 15;
        bad += ((word >> k) & 1u) != ((row[r] >> e) & 1u);
        bad += ((word >> (16 + k)) & 1u) != ((row[r] >> (16 + e)) & 1u);
      }
    }
  }
  return bad;
}

static int type_faults() {
  int bad = 0;
  for (int type = 0; type < 4096; ++type)
    for (int code = 0; code < 8; ++code) {   // region 0-3, cluster
      const int t = type | (code & 3) << kRegionShift | (code >> 2) << 30;
      bad += type_word(type_half(t)) != t;
    }
  return bad;
}

int main() {
  std::mt19937_64 rng(5);
  std::printf("%.6f %d %d\n", step_error(rng), order_faults(rng), type_faults());
  return 0;
}
"""


@pytest.fixture(scope="module")
def figures(tmp_path_factory):
    if shutil.which(build.nvcc()) is None:
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("arith")
    src, exe = d / "arith.cu", d / "arith"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-I" + os.path.join(build.ROOT, "include"),
                    "-I" + build.CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    return float(out[0]), int(out[1]), int(out[2])


def test_rsqrt_step(figures):
    """Result's rounding 1, that of 1 - x y^2 half, the step's own 5/16 (2^-19)^3: 1.52 x 2^-53."""
    assert figures[0] < 1.53


def test_record_bit_orders(figures):
    assert figures[1] == 0


def test_type_words(figures):
    assert figures[2] == 0
