"""The FP64 form's division by a known divisor (csrc/div_by.cuh) equals the
IEEE division in every way it can take: divisors of every kind (1, powers of
two, short, general, out of range, special), and numerators that put the
quotient next to a rounding boundary (x 2^t = s mod Y for small s, by modular
inversion), next to a representable value, at zero, at the ends of the range
and beyond."""
import math
import random
import struct
import subprocess

import pytest


def hard_numerators(y, rnd):
    """x whose quotient by y lies within a few units of the remainder of a boundary."""
    Y = int(math.ldexp(math.frexp(y)[0], 53))
    odd = Y
    while odd % 2 == 0:
        odd //= 2
    out = []
    if odd > 1:
        for s in (1, -1, 2, -2, 3, -3):
            for t in (52, 53, 54, 55):
                X = s * pow(pow(2, t, odd), -1, odd) % odd
                while 0 < X < 2 ** 52:
                    X *= 2
                if 0 < X < 2 ** 53:
                    out.append(math.ldexp(X, -53) * rnd.choice((1.0, -1.0, 2.0 ** -40, 2.0 ** 9)))
    return out


def pairs():
    rnd = random.Random(3)
    ys = [1.0, 2.0, 0.5, 0.25, 3.0, 5.0, 10.0, 0.75, 0.7, 0.8, 0.52, 0.6, 0.55, 1.0 - 2 ** -53, 1.0 + 2 ** -52, 2.0 - 2 ** -52]
    ys += [rnd.uniform(0.5, 2.0) for _ in range(1500)]
    ys += [0.5 + rnd.uniform(0.0, 3.0) * 10.0 ** -rnd.randint(0, 9) for _ in range(1500)]
    for y in ys:
        for x in hard_numerators(y, rnd):
            yield x, y
        for _ in range(20):
            x = rnd.uniform(0.5, 1.0) * y
            yield from ((x, y), (math.nextafter(x, 0.0), y), (rnd.uniform(-1.0, 1.0) * 10.0 ** -rnd.randint(0, 17), y))
        for x in (0.0, -0.0, 5e-324, 1e-310, 1.7e308, math.inf, -math.inf, math.nan, 2.0 ** -823, 2.0 ** -824,
                  2.0 ** 777, math.nextafter(2.0 ** 777, 0.0)):
            yield x, y
    for y in (1e-200, 1e200, 2.0 ** -101, -0.7, 0.0, math.inf, math.nan, 5e-324):
        for x in (1.0, -3.0, 0.0, 1e-300, math.inf, math.nan):
            yield x, y


def test_div_by_equals_ieee_division(tmp_path):
    exe, data = tmp_path / "div_by_check", tmp_path / "pairs.bin"
    r = subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-o", str(exe), "tests/c/div_by_check.cpp"],
                       capture_output=True, text=True)
    if r.returncode:
        pytest.fail(r.stderr)
    data.write_bytes(b"".join(struct.pack("<dd", x, y) for x, y in pairs()))
    n, bad, *how = (int(v) for v in subprocess.run([str(exe), str(data)], capture_output=True, text=True,
                                                   check=True).stdout.split())
    assert n > 100000 and min(how) > 0, (n, how)
    assert bad == 0
