// div_by_check -- div_by (droplet_gb300/csrc/div_by.cuh) against the machine's
// IEEE division on pairs (x, y) of doubles read from the file argv[1]. Prints
// the number of pairs, of quotients that differ (zeros compare equal whatever
// their sign, NaN equals NaN), and how many pairs took each way.
#include "../../droplet_gb300/csrc/div_by.cuh"

#include <stdio.h>

using namespace dl;

static bool same(double a, double b) { return a == b || (a != a && b != b); }

int main(int argc, char** argv) {
    FILE* f = argc > 1 ? fopen(argv[1], "rb") : nullptr;
    if (!f) return 2;
    long n = 0, bad = 0, how[6] = {0, 0, 0, 0, 0, 0};
    double v[2];
    while (fread(v, sizeof(double), 2, f) == 2) {
        const volatile double x = v[0], y = v[1];
        const double want = x / y;
        const DivBy d = make_div_by(v[1]);
        how[d.how] += 1;
        bad += !same(div_by(v[0], d), want);
        // the way of a divisor that only the device knows
        if (div_divisor_ok(v[1]) && div_numerator_ok(v[0])) {
            const double zh = 1.0 / v[1];
            bad += !same(div_correct(v[0], v[1], zh, div_fma(-v[1], zh, 1.0) * zh), want);
        }
        ++n;
    }
    fclose(f);
    printf("%ld %ld %ld %ld %ld %ld %ld %ld\n", n, bad, how[0], how[1], how[2], how[3], how[4], how[5]);
    return 0;
}
