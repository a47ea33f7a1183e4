// The fit's division by a shared reciprocal (div_by, csrc/at_device.cuh) on the
// host against the division it stands for, bit for bit, over the ranges that
// its moments have.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include "../apriltags_fast_b200/csrc/at_device.cuh"

static uint64_t state = 88172645463325252ull;
static uint64_t next() {
    state ^= state << 13;
    state ^= state >> 7;
    return state ^= state << 17;
}
// A double of exponent e: a mantissa drawn, or of few ones, or nearly all ones.
static double draw(int e) {
    uint64_t m = next() & 0xfffffffffffffull;
    switch (next() & 7) {
    case 0: m = next() & 3; break;
    case 1: m = 0xfffffffffffffull - (next() & 3); break;
    case 2: m = ~0ull << (next() % 52) & 0xfffffffffffffull; break;
    case 3: m &= ~0ull << (next() % 52); break;
    }
    const uint64_t b = (uint64_t)(e + 1023) << 52 | m;
    double d;
    memcpy(&d, &b, 8);
    return d;
}

int main() {
    long bad = 0;
    auto check = [&](double a, double b) {
        const double want = a / b, got = div_by(a, b, 1.0 / b);
        if (memcmp(&want, &got, 8) && bad++ < 10) printf("%a / %a: %a, not %a\n", a, b, got, want);
    };
    for (long n = 0; n < 4000000; n++) {
        const double b = draw((int)(next() % 27) - 1);
        check(0.0, b);
        const double a = draw((int)(next() % 111) - 54);
        check(a, b);
        check(-a, b);
        // quotients at, and next to, a value and the middle of two
        const double q = draw((int)(next() % 57) - 30), p = q * b, h = fma(q, b, 0x1p-53 * q * b);
        for (double x : {p, nextafter(p, 0.0), nextafter(p, 1e300), h, nextafter(h, 0.0), nextafter(h, 1e300)}) check(x, b);
    }
    printf("%ld differ\n", bad);
    return bad != 0;
}
