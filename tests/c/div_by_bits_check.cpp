// div_by_bits_check -- div_by (droplet_gb300/csrc/div_by.cuh) against the machine's
// IEEE division by bit pattern (the signs of zeros included; NaN equals NaN) on
// pairs (x, y) of doubles read from the file argv[1]. Prints the number of pairs,
// of zero numerators among them, and of quotients that differ.
#include "../../droplet_gb300/csrc/div_by.cuh"

#include <stdio.h>

using namespace dl;

static bool same(double a, double b) { return div_bits(a) == div_bits(b) || (a != a && b != b); }

int main(int argc, char** argv) {
    FILE* f = argc > 1 ? fopen(argv[1], "rb") : nullptr;
    if (!f) return 2;
    long n = 0, zeros = 0, bad = 0;
    double v[2];
    while (fread(v, sizeof(double), 2, f) == 2) {
        const volatile double x = v[0], y = v[1];
        const double want = x / y;
        bad += !same(div_by(v[0], make_div_by(v[1])), want);
        if (div_divisor_ok(v[1]) && div_numerator_ok(v[0])) {  // the way of a divisor that only the device knows
            const double zh = 1.0 / v[1];
            bad += !same(div_correct(v[0], v[1], zh, div_fma(-v[1], zh, 1.0) * zh), want);
        }
        zeros += v[0] == 0.0;
        ++n;
    }
    fclose(f);
    printf("%ld %ld %ld\n", n, zeros, bad);
    return 0;
}
