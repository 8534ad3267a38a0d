"""The quotient of the grid lookups (csrc/rgpu_quotient.h) against the division, compiled for the host: random
operands and, for random divisors B, the numerators whose quotient comes closest to the middle between two doubles
(M * B = +-1 modulo 2^54 for the odd 54-bit number M of that middle)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "raspa2_b200", "csrc")

PROGRAM = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include "rgpu_quotient.h"
static uint64_t s = 88172645463325252ULL;
static uint64_t rnd(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static long tried, differ;
static void check(double x, double b) { tried++; differ += rgpu_quotient(x, b, 1.0 / b) != x / b; }
int main(void)
{
  for (long i = 0; i < 4000000; i++) {
    /* mantissas: random, just above a power of two, just below one */
    uint64_t B = (rnd() >> 12) | 1ULL << 52 | 1;
    if (i % 4 == 1) B = 1ULL << 52 | (rnd() & 0xfffff) | 1;
    if (i % 4 == 2) B = (1ULL << 53) - 1 - (rnd() & 0xffffe);
    check(ldexp((double)((rnd() >> 12) | 1ULL << 52), (int)(rnd() % 80) - 100), ldexp((double)B, (int)(rnd() % 80) - 100));
    uint64_t inv = B;
    for (int k = 0; k < 6; k++) inv *= 2 - B * inv;
    for (int sign = 0; sign < 2; sign++) {
      const uint64_t M = (sign ? inv : 0 - inv) & ((1ULL << 54) - 1);
      const uint64_t X = (uint64_t)(((unsigned __int128)M * B + (sign ? -1 : 1)) >> 54);
      if (M >> 53 && X >> 52 && (uint64_t)(double)X == X) check((double)X, (double)B);
    }
  }
  printf("%ld %ld\n", tried, differ);
  return 0;
}
"""


def test_quotient_rounds_as_the_division(tmp_path):
    gcc = shutil.which("gcc")
    if not gcc:
        pytest.skip("no C compiler")
    (tmp_path / "q.c").write_text(PROGRAM)
    exe = str(tmp_path / "q")
    subprocess.check_call([gcc, "-O2", "-ffp-contract=off", "-D__host__=", "-D__device__=", "-I" + CSRC, "-o", exe,
                           str(tmp_path / "q.c"), "-lm"])
    tried, differ = map(int, subprocess.check_output([exe]).split())
    assert tried > 5_000_000 and differ == 0
