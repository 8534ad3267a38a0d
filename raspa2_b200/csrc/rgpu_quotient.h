/* Quotients by a divisor whose reciprocal is kept. */
#ifndef RGPU_QUOTIENT_H
#define RGPU_QUOTIENT_H

#include <math.h>

/* x / b from ib = 1 / b (rounded): the product x * ib, which is within 1.5
 * units in the last place, and one residual correction (Markstein,
 * "Computation of elementary functions on the IBM RISC System/6000 processor",
 * 1990). The result is within 0.5 + 2^-51 units of x / b, so it is one of the
 * two doubles about it and, unless x / b lies within 2^-51 units of the middle
 * between two, the division's result (the theorem there, which has no
 * exception, asks for a first quotient within one unit). No exception was
 * found among random operands and the quotients closest to a middle
 * (test_quotient.py). For x and quotients in the range of normal numbers. A
 * third of a division's instructions. */
__host__ __device__ inline double rgpu_quotient(double x, double b, double ib)
{
  const double q = x * ib;
  return fma(fma(-q, b, x), ib, q);
}

#endif
