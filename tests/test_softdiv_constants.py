"""Multiples by 3, 5, 7 and 11 on the integer pipes (csrc/softdiv.cuh mulc)
against IEEE multiplication, on the host."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "hamstr_oop_gb300", "csrc")

PROGRAM = r"""
#include "softdiv.cuh"
#include <cstdio>
#include <random>
using namespace hamstr::sd;
int main() {
   std::mt19937_64 rng(23);
   long bad = 0, n = 0;
   for (long i = 0; i < 8000000; i++) {
      uint64_t u = rng();
      const int mode = (int)(i % 8);
      if (mode == 0) u = (u & 0xFFF00000000000FFull);                                      // few bits set
      if (mode == 1) u = u | 0xFFFFFFFFFFF00ull;                                           // all but the last ones
      if (mode == 2) u = (u & 0x800FFFFFFFFFFFFFull) | (0x7FEull - rng() % 6) << 52;       // near overflow
      if (mode == 3) u = (u & 0x800FFFFFFFFFFFFFull) | (rng() % 3) << 52;                  // subnormal and just above
      if (mode == 4) u = (u & 0x8000000000000000ull) | ((rng() & 1) ? 0x7FF0000000000000ull : 0);   // inf, zero
      if (mode == 5) u = (u & 0x800FFFFFFFFFFFFFull) | (1000 + rng() % 46) << 52;
      const double x = from_bits(u);
      const double w[4] = {x * 3., x * 5., x * 7., x * 11.}, g[4] = {mulc<3>(x), mulc<5>(x), mulc<7>(x), mulc<11>(x)};
      for (int k = 0; k < 4; k++) {
         n++;
         if (bits(w[k]) != bits(g[k]) && !(w[k] != w[k] && g[k] != g[k])) bad++;
      }
   }
   printf("%ld %ld\n", bad, n);
   return bad != 0;
}
"""


def test_small_multiples_match_the_multiply_on_the_host(tmp_path):
    src = tmp_path / "c.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "c"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    bad, n = (int(x) for x in out.stdout.split())
    assert out.returncode == 0 and bad == 0 and n == 32000000
