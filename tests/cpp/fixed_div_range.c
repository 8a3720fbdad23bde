/* Host check of the fixed-divisor division sequence (see fixed_div_check.c) for smoothing
 * lengths h from 2^-24 to 2^20 and their squares: verified on one binade, it gives the IEEE
 * quotient for every dividend of magnitude in [2^-100, 2^100] whose quotient is normal.
 * Prints "ok <divisors> <dividends>" or the first counterexample. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

static float f_of(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }

static float seq(float a, float b, float y) {
    const float q0 = a * y;
    const float r = fmaf(-q0, b, a);
    return fmaf(r, y, q0);
}

static uint64_t state = 1;
static uint64_t next(void) {  /* splitmix64 */
    uint64_t z = (state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

int main(void) {
    int divisors = 0;
    long tested = 0;
    for (int k = 0; k < 45; ++k) {
        /* 2^-24 .. 2^20, the ends exactly, random significands between them */
        const float sig = k == 0 || k == 44 ? 1.0f : f_of(0x3f800000u | (uint32_t)(next() >> 41));
        const float h = ldexpf(sig, k - 24);
        for (int sq = 0; sq < 2; ++sq) {
            const float b = sq ? h * h : h, y = 1.0f / b;
            int ok = 1;
            for (uint32_t m = 0; m < (1u << 23) && ok; ++m) {
                const float a = f_of(0x3f800000u | m);
                ok = seq(a, b, y) == a / b;
            }
            if (!ok) continue;
            ++divisors;
            for (int i = 0; i < (1 << 17); ++i) {
                const uint64_t z = next();
                const int e = (int)(z % 201) - 100;
                const float a = f_of((uint32_t)(z >> 63) << 31 | (uint32_t)(127 + e) << 23 |
                                     ((uint32_t)(z >> 20) & 0x7fffffu));
                const float want = a / b;
                if (fabsf(want) < 0x1p-126f || fabsf(want) > 0x1p127f) continue;
                ++tested;
                if (seq(a, b, y) != want) {
                    printf("mismatch b=%a a=%a\n", b, a);
                    return 1;
                }
            }
        }
    }
    printf("ok %d %ld\n", divisors, tested);
    return 0;
}
