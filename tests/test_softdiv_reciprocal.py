"""The integer-pipe reciprocal (csrc/softdiv.cuh recip64, rcp) against exact
integers and IEEE division.

recip64 gives 2^64/m from an FP32 estimate of 1/m; the rounding of every
quotient rests on its error bounds, which must hold for any estimate within
1.5 * 2^-23 of the reciprocal, relative (the device's approximate reciprocal differs from the host's in the
last place).  The header is compiled with the host compiler."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "hamstr_oop_gb300", "csrc")

PROGRAM = r"""
#include "softdiv.cuh"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace hamstr::sd;
int main(int, char** argv) {
   const int ulps = atoi(argv[1]);   // moves the seed that many FP32 places
   std::mt19937_64 rng(17);
   long bad = 0, n = 0;
   for (long i = 0; i < 4000000; i++) {
      uint64_t m = rng() & 0xFFFFFFFFFFFFFull;
      const int k = (int)(i % 8);
      if (k == 0) m = i / 8 < 256 ? i / 8 : rng() & 0xFF;                    // at and just above a power of two
      if (k == 1) m = 0xFFFFFFFFFFFFFull - (rng() & 0xFF);
      if (k == 2) m = (rng() & 0x7FFFFF) << 29;                              // the estimate's own 24 bits
      if (k == 3) m = ((rng() & 0x7FFFFF) << 29) | 0x1FFFFFFF;
      const uint64_t mb = m | 0x10000000000000ull;
      float y = recip_seed(mb);
      for (int t = 0; t < abs(ulps); t++) y = nextafterf(y, ulps < 0 ? 0.f : 2.f);
      const uint64_t r = recip64(mb, y);
      const unsigned __int128 one = (unsigned __int128)1 << 116;             // 2^64 / m = 2^116 / mb
      const __int128 below = (__int128)(one / mb) - (__int128)r;             // floor(true) - r
      if (below < 0 || below > 7) bad++;
      n++;
      int e = 1 + (int)(rng() % 2046);
      if (i % 3) e = 1000 + (int)(rng() % 46);
      const double b = from_bits((rng() & 0x8000000000000000ull) | ((uint64_t)e << 52) | m), w = 1.0 / b, g = rcp(b);
      if (bits(w) != bits(g)) bad++;
   }
   const double other[] = {0.0, -0.0, 4.9e-324, -2.2e-308, 1.7976931348623157e308, -8.9e307, 4.49e307,
                           from_bits(0x7FF0000000000000ull), from_bits(0xFFF0000000000000ull)};
   for (double b : other) {
      n++;
      if (bits(1.0 / b) != bits(rcp(b))) bad++;
   }
   if (rcp(from_bits(0x7FF8000000000000ull)) == rcp(from_bits(0x7FF8000000000000ull))) bad++;
   printf("%ld %ld\n", bad, n);
   return bad != 0;
}
"""


@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_reciprocal_bounds_and_rounding_on_the_host(tmp_path, ulps):
    src = tmp_path / "r.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "r"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(ulps)], capture_output=True, text=True)
    bad, n = (int(x) for x in out.stdout.split())
    assert out.returncode == 0 and bad == 0 and n == 4000009
