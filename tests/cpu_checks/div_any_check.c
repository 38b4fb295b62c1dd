/* Checks that dividing by any b through y = RN(1/b) with two corrections,
 *   q = RN(a*y); q = RN(q + RN(a - q*b) * y), twice,
 * gives the IEEE quotient, for the dividends and divisors of the frontend's Y
 * reconstruction (an integer quantum times a weight, over a quantiser scale):
 * divisors over the whole significand range, among them the first and last
 * ones, dividends random and at the quotients hardest to round (a = RN(b * m)
 * for midpoints m of adjacent floats, and its neighbours). Prints the number of
 * quotients that differ and exits non-zero if there are any. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

static float from_bits(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}
static uint32_t to_bits(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}
static uint64_t state = 0x9e3779b97f4a7c15ull;
static uint32_t next(void) {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return (uint32_t)(state >> 32);
}
static int differs(float a, float b) {
    const float y = 1.0f / b;
    float q = a * y;
    q = fmaf(fmaf(q, -b, a), y, q);
    q = fmaf(fmaf(q, -b, a), y, q);
    return q != a / b;
}

int main(void) {
    long long bad = 0, total = 0;
    for (int i = 0; i < 60000; ++i) {
        /* b in [2^-8, 2^8): the scales are qf / 65536 * gs. */
        uint32_t m = i < 64 ? (uint32_t)i : (i < 128 ? 0x7fffffu - (uint32_t)(i - 64) : next() & 0x7fffffu);
        const float b = from_bits(((119u + next() % 16u) << 23) | m);
        for (int k = 0; k < 2000; ++k) {
            float a;
            if (k & 1) {
                const float q = from_bits(((110u + next() % 30u) << 23) | (next() & 0x7fffffu));
                const double mid = 0.5 * ((double)q + (double)from_bits(to_bits(q) + 1));
                a = (float)(mid * (double)b);
                a = from_bits(to_bits(a) + next() % 3u - 1u);
            } else {
                a = (float)(1 + next() % 32768u) * from_bits(((112u + next() % 16u) << 23) | (next() & 0x7fffffu));
            }
            ++total;
            bad += differs(a, b);
        }
    }
    bad += differs(0.0f, 0.37f);
    printf("%lld quotients, %lld mismatching\n", total, bad);
    return bad != 0;
}
