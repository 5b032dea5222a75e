// split2_f64 / split3_f64 (meshoid_gb300/csrc/mg_split.cuh) against the FP64
// expressions they stand for, bit for bit: random significands at every
// exponent, values on and beside the rounding boundaries, and the special ones.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../meshoid_gb300/csrc/mg_split.cuh"

static long bad = 0, done = 0;

static bool same(float a, float b) {
    uint32_t x, y;
    memcpy(&x, &a, 4);
    memcpy(&y, &b, 4);
    return x == y || (a != a && b != b) || (a == 0.0f && b == 0.0f);
}

static void check(double v) {
    const float h = (float)v;
    const double r = v - (double)h;
    const float m = (float)r, l = (float)(r - (double)m);
    float a, b, c, d, e;
    mg::split2_f64(v, a, b);
    mg::split3_f64(v, c, d, e);
    ++done;
    if (!same(a, h) || !same(b, m) || !same(c, h) || !same(d, m) || !same(e, l)) {
        if (bad++ < 10) printf("%a: %a %a | %a %a %a, want %a %a %a\n", v, a, b, c, d, e, h, m, l);
    }
}

int main() {
    std::mt19937_64 g(7);
    for (uint64_t ex = 0; ex < 2048; ++ex)
        for (int i = 0; i < 4000; ++i) {
            uint64_t m = g() & 0xfffffffffffffull;
            switch (i % 8) {
                case 0: m = (m & ~0x1fffffffull) | 0x10000000ull; break;            // a tie
                case 1: m = (m & ~0x1fffffffull) | 0x10000001ull; break;            // just above
                case 2: m = (m & ~0x1fffffffull) | 0x0fffffffull; break;            // just below
                case 3: m |= 0xfffffff000000ull; break;                             // carries
                case 4: m &= ~0x1fffffffull; break;                                 // exact
                case 5: m = (m & ~0x1fffffffull) | (g() & 31u); break;              // short remainder
                default: break;
            }
            const uint64_t b = (g() & 1ull) << 63 | ex << 52 | m;
            double v;
            memcpy(&v, &b, 8);
            check(v);
        }
    const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 1.0, -1.0, 3.4028235677973366e38, 1e300, 5e-324};
    for (double v : special) check(v);
    printf("%ld values, %ld differ\n%s\n", done, bad, bad ? "FAILED" : "ok");
    return bad ? 1 : 0;
}
