"""Products and quotients of a doubled operand on the integer pipes
(csrc/softdiv.cuh mul<K>, div<K>) against the operators, bit for bit, over
the whole range: a doubling that overflows, subnormal operands and results,
zeros, infinities.  The header is compiled with the host compiler."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "hamstr_oop_gb300", "csrc")

PROGRAM = r"""
#include "softdiv.cuh"
#include <cstdio>
#include <random>
using namespace hamstr::sd;
static std::mt19937_64 rng(23);
static double draw(int kind) {
   const uint64_t r = rng(), m = r & 0xFFFFFFFFFFFFFull, sign = r & 0x8000000000000000ull;
   const uint64_t e = kind == 0 ? 1000 + rng() % 47 : kind == 1 ? rng() % 3 : kind == 2 ? 2043 + rng() % 5 : rng() % 2048;
   return from_bits(sign | (e << 52) | (e >= 2047 || rng() % 16 == 0 ? 0 : m));
}
static bool same(double x, double y) { return bits(x) == bits(y) || (x != x && y != y); }
int main() {
   long bad = 0, n = 0;
   for (long i = 0; i < 3000000; i++) {
      const double a = draw(i % 4), b = draw((i / 4) % 4);
      bad += !same(mul<1>(a, b), (2.0 * a) * b) + !same(div<1>(a, divisor(b)), (2.0 * a) / b);
      bad += !same(mul<0>(a, b), a * b) + !same(div<0>(a, divisor(b)), a / b);
      n += 4;
   }
   printf("%ld %ld\n", bad, n);
   return bad != 0;
}
"""


def test_doubled_operands_match_the_operators(tmp_path):
    src = tmp_path / "scaled.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "scaled"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    bad, n = (int(x) for x in r.stdout.split())
    assert n == 12000000 and bad == 0
