/* The square root, reciprocal and quotients of csrc/voxel.cuh's shrink_rn against the IEEE
 * operations: l = RN(sqrt(s)) for every s in [1, 4) and every reciprocal square root within 2 ulp
 * (larger s are these times a power of four); r = RN(1 / l) but for the few l that are counted;
 * the same step from a reciprocal of any b within 1 ulp; RN(a / l) by two corrections, for these l over every numerator of two binades, and for random
 * operands, ends of a binade among them, over the range 1 <= l <= 2^20, a zero or at least 2^-60.
 * Prints what differs (other than in the sign of a zero). */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static uint64_t state = 88172645463325252ull;
static uint64_t next(void)
{
    state ^= state << 13, state ^= state >> 7, state ^= state << 17;
    return state;
}
static float bits(uint32_t b)
{
    float f;
    memcpy(&f, &b, 4);
    return f;
}
static uint32_t bits_of(float f)
{
    uint32_t b;
    memcpy(&b, &f, 4);
    return b;
}

static void root(float s, float y, float *l, float *r)
{
    float g = s * y, h = 0.5f * y;
    const float e = fmaf(-g, h, 0.5f);
    g = fmaf(g, e, g);
    h = fmaf(h, e, h);
    *l = fmaf(fmaf(-g, g, s), h, g);
    const float t = h + h;
    const float f = fmaf(-*l, t, 1.0f);
    *r = fmaf(fmaf(f + f, f, f), t, t);
}

static long quotient(float a, float l, float r)
{
    float q = a * r;
    q = fmaf(fmaf(-l, q, a), r, q);
    q = fmaf(fmaf(-l, q, a), r, q);
    if (q == a / l) return 0;
    printf("%a / %a by %a: %a, not %a\n", a, l, r, q, a / l);
    return 1;
}

int main(int argc, char **argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 4000000;
    long bad = 0, inexact = 0;
    float l_done = 0.0f, r_done = 0.0f;
    for (uint32_t i = 0x3f800000u; i < 0x40800000u && bad < 20; ++i) {
        const float s = bits(i);
        const uint32_t y0 = bits_of((float)(1.0 / sqrt((double)s)));
        for (int d = -2; d <= 2; ++d) {
            float l, r;
            root(s, bits(y0 + (uint32_t)d), &l, &r);
            if (l != sqrtf(s)) printf("sqrt(%a): %a\n", s, l), ++bad;
            if (r == 1.0f / l || (l == l_done && r == r_done)) continue;
            ++inexact;
            l_done = l, r_done = r;
            for (uint32_t m = 0x3f800000u; m < 0x40800000u && bad < 20; ++m) bad += quotient(bits(m), l, r);
        }
    }
    /* the same step from a reciprocal within 1 ulp, for every divisor's mantissa */
    for (uint32_t i = 0x3f800000u; i < 0x40000000u && bad < 20; ++i) {
        const float b = bits(i);
        for (int d = -1; d <= 1; ++d) {
            const float t = bits(bits_of(1.0f / b) + (uint32_t)d);
            const float f = fmaf(-b, t, 1.0f), r = fmaf(fmaf(f + f, f, f), t, t);
            if (r == 1.0f / b || (b == l_done && r == r_done)) continue;
            ++inexact;
            l_done = b, r_done = r;
            for (uint32_t m = 0x3f800000u; m < 0x40800000u && bad < 20; ++m) bad += quotient(bits(m), b, r);
        }
    }
    for (long i = 0; i < n && bad < 20; ++i) {
        const uint64_t x = next(), y = next();
        const float a = bits((uint32_t)((x >> 63) << 31) | (uint32_t)(67 + (x >> 32) % 101) << 23 |
                             (uint32_t)(x & 0x7fffff));
        const float b = bits((uint32_t)(127 + (y >> 32) % 20) << 23 | (uint32_t)(y & 0x7fffff));
        const float ae = bits((uint32_t)(127 + (x >> 40) % 3) << 23 | ((x & 1) ? 0x7fffff - (uint32_t)(x >> 50) % 64
                                                                              : (uint32_t)(x >> 50) % 64));
        const float be = bits((uint32_t)(127 + (y >> 40) % 3) << 23 | ((y & 1) ? 0x7fffff - (uint32_t)(y >> 50) % 64
                                                                              : (uint32_t)(y >> 50) % 64));
        bad += quotient(a, b, 1.0f / b) + quotient(ae, b, 1.0f / b) + quotient(a, be, 1.0f / be) +
               quotient(ae, be, 1.0f / be) + quotient(0.0f, b, 1.0f / b);
    }
    printf("%ld inexact reciprocals, %ld differ\n", inexact, bad);
    return bad != 0;
}
