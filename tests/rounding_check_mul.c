/* The float forms of double-precision steps that the encode kernel relies on
 * (h261enc_cuda_b200/csrc/kernels.cu), checked on the CPU:
 *
 * 1. mul_hilo: (float)((double)x * k) == fmaf(x, hi, x * lo), hi = (float)k,
 *    lo = (float)(k - hi), for every mantissa x in [1, 2) (products scale by
 *    powers of two, and a sign changes both sides alike).  0.382683 and
 *    1.84776: every mantissa.  0.707107: every one of at most 18 significant
 *    bits, which covers the integers below 2^18 that the first pass of the
 *    forward DCT multiplies.
 * 2. idct_round: floor((double)v + 0.49999) == floor of v + 0.49999f rounded
 *    down to float, for every float of magnitude 2^-25 .. 2^18.  Both sides
 *    grow with v and are 0 at +-2^-25, so they are 0 in between.
 *
 * Built and run by tests/test_rounding_mul.py; prints the count of checks
 * and of differences. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

static float bits(uint32_t u)
{
    float x;
    memcpy(&x, &u, sizeof(x));
    return x;
}

static long checked, differing;

static void mul(double k, uint32_t step)
{
    const float hi = (float)k, lo = (float)(k - (double)hi);
    for (uint32_t u = 0x3f800000u; u < 0x40000000u; u += step) {
        const float x = bits(u);
        checked++;
        differing += (float)((double)x * k) != fmaf(x, hi, x * lo);
    }
}

int main(void)
{
    mul(0.382683, 1);
    mul(1.84776, 1);
    mul(0.707107, 1u << 6);   /* 24 - 6 = 18 significant bits */
    for (uint32_t u = 0x33000000u; u < 0x48800000u; u++)
        for (int sign = 0; sign < 2; sign++) {
            const float v = sign ? -bits(u) : bits(u);
            const double sum = (double)v + (double)0.49999f;   /* exact: under 53 bits apart */
            float down = (float)sum;
            if ((double)down > sum)
                down = nextafterf(down, -INFINITY);
            checked++;
            differing += floor((double)v + 0.49999) != (double)floorf(down);
        }
    printf("%ld %ld\n", checked, differing);
    return differing != 0;
}
