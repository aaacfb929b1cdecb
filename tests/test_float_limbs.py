"""FP32 values as integers over a common exponent (the gradient's block sums; CPU)."""
import os
import subprocess
from fractions import Fraction

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cylinder-flow_gb300", "csrc")

PROG = r"""
#include <cstdio>
#include <cstring>
#include <cstdint>
#include "float_limbs.hpp"
// 128 floats (bits) a line: e and the three sums
int main() {
  uint32_t b[128];
  while (true) {
    uint32_t top = 0;
    for (int k = 0; k < 128; ++k) {
      if (std::scanf("%u", &b[k]) != 1) return 0;
      if ((b[k] & 0x7FFFFFFFu) > top) top = b[k] & 0x7FFFFFFFu;
    }
    const int e = (int)(top >> 23);
    const uint32_t sbits = (uint32_t)(276 - e) << 23;
    float scale, v;
    std::memcpy(&scale, &sbits, 4);
    int s[3] = {0, 0, 0};
    for (int k = 0; k < 128; ++k) {
      std::memcpy(&v, &b[k], 4);
      const cflbm::FloatLimbs l = cflbm::float_limbs(v, scale);
      if (__builtin_add_overflow(s[0], l.a, &s[0]) || __builtin_add_overflow(s[1], l.b, &s[1]) ||
          __builtin_add_overflow(s[2], l.c, &s[2])) return 1;
    }
    std::printf("%d %d %d %d\n", e, s[0], s[1], s[2]);
  }
}
"""


def blocks():
    rng = np.random.default_rng(4)
    for decades in (0, 3, 12, 30):
        for size in (1e-24, 1.0, 1e30):
            yield (rng.normal(size=128) * size * 10.0 ** -rng.uniform(0, decades, 128)).astype(np.float32)
    yield np.full(128, np.float32(np.finfo(np.float32).max))          # largest sums
    yield np.full(128, -np.nextafter(np.float32(2), np.float32(0)))
    yield np.where(np.arange(128) % 2, 1, -1 + 2.0 ** -24).astype(np.float32)  # cancellation
    yield np.array([1.0] + [2.0 ** -60] * 127, np.float32)            # far below 2^-53 of the largest


def test_block_sums_at_least_as_accurate_as_fp64(tmp_path):
    (tmp_path / "p.cpp").write_text(PROG)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")], check=True)
    bs = list(blocks())
    text = "\n".join(" ".join(map(str, b.view(np.uint32))) for b in bs)
    out = subprocess.run([str(tmp_path / "p")], input=text, text=True, capture_output=True, check=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) == len(bs)
    for b, (e, sa, sb, sc) in zip(bs, rows):
        exact = sum(Fraction(float(v)) for v in b)
        got = (Fraction(sa) + Fraction(sb, 2 ** 24) + Fraction(sc, 2 ** 48)) * Fraction(2) ** (e - 149)
        assert abs(got - exact) <= 128 * Fraction(2) ** (e - 126 - 72)
        # rounded once to FP64, against additions one by one
        total = 0.0
        for v in b:
            total += float(v)
        assert abs(Fraction(float(got)) - exact) <= abs(Fraction(total) - exact) + abs(exact) * Fraction(2) ** -53
