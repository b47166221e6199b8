// Host check of fp64_alu.cuh: divisions and square roots against the host's
// IEEE operations over random and edge operands.  argv[1]: pairs to draw.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "../gpueularsolver2d_gb300/csrc/fp64_alu.cuh"

static uint64_t st = 88172645463325252ULL;
static uint64_t rnd() {
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st;
}

static bool same(double a, double b) {
    return e2d::bits_of(a) == e2d::bits_of(b) || (a != a && b != b);
}

static uint64_t draw_significand(int kind) {
    const uint64_t all = 0xFFFFFFFFFFFFFULL;
    switch (kind) {
        case 0: return rnd() & all;
        case 1: return rnd() & 7;                                // just above a power of two
        case 2: return all - (rnd() & 7);                        // just below one
        case 3: return (rnd() & 0x7fffffULL) << 29;              // exact in the seed's 24 bits
        case 4: return (((rnd() & 0x7fffffULL) << 29) - 1) & all;  // the seed's truncation at its largest
        default: return (rnd() & rnd() & rnd()) & all;           // few bits set
    }
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    const double special[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 5e-324, 2.2250738585072014e-308,
                              1.7976931348623157e308, 2.2250738585072009e-308, 3.0, 4.0, 0.1, 1e-300, 1e300};
    long bad = 0;
    auto check = [&](double a, double b) {
        if (!same(e2d::ddiv(a, b), a / b)) {
            if (bad++ < 5) printf("div %a %a: %a, not %a\n", a, b, e2d::ddiv(a, b), a / b);
        }
        if (!same(e2d::dsqrt(a), std::sqrt(a))) {
            if (bad++ < 5) printf("sqrt %a: %a, not %a\n", a, e2d::dsqrt(a), std::sqrt(a));
        }
        if (!same(e2d::imul(a, b), a * b)) {
            if (bad++ < 5) printf("mul %a %a: %a, not %a\n", a, b, e2d::imul(a, b), a * b);
        }
        const bool lt = e2d::order_key(a) < e2d::order_key(b);
        if (a == a && b == b && a != b && lt != (a < b)) bad++;
        if (!same(e2d::key_value(e2d::order_key(a)), a)) bad++;
    };
    for (double a : special)
        for (double b : special) check(a, b);
    for (long k = 0; k < n; k++) {
        const uint64_t r = rnd();
        // exponents near one another, and now and then over the whole range
        const uint64_t ea = (r & 15) ? 1003 + (r >> 8) % 41 : (r >> 8) & 0x7ff;
        const uint64_t eb = (r & 15) ? 1003 + (r >> 20) % 41 : (r >> 20) & 0x7ff;
        const double a = e2d::double_of((r & 0x8000000000000000ULL) | (ea << 52) | draw_significand((r >> 40) % 6));
        const double b = e2d::double_of(((r << 1) & 0x8000000000000000ULL) | (eb << 52) | draw_significand((r >> 44) % 6));
        check(a, b);
        check(std::fabs(b), a);
        check(a * b, b);  // quotients close to representable numbers
        check(a * a, a);
        // products half way between two numbers, and next to it
        const uint64_t odd = (rnd() & 0x3ffffff) | 1, big = (1ULL << 52) | (rnd() & 0xFFFFFFFFFFFFFULL);
        check((double)(odd | 0x4000000), (double)(rnd() & 0x7ffffff));
        check((double)big, (double)(odd & 7));
    }
    printf("%ld\n", bad);
    return bad != 0;
}
