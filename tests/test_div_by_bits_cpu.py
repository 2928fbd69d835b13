"""The division of csrc/div_by.cuh has the IEEE division's bits, the sign of a zero
quotient included, on the pairs of test_div_by_cpu.py (every divisor there meets
both zeros)."""
import struct
import subprocess

import pytest

from test_div_by_cpu import pairs


def test_div_by_has_the_bits_of_ieee_division(tmp_path):
    exe, data = tmp_path / "div_by_bits_check", tmp_path / "pairs.bin"
    r = subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-o", str(exe), "tests/c/div_by_bits_check.cpp"],
                       capture_output=True, text=True)
    if r.returncode:
        pytest.fail(r.stderr)
    data.write_bytes(b"".join(struct.pack("<dd", x, y) for x, y in pairs()))
    n, zeros, bad = (int(v) for v in subprocess.run([str(exe), str(data)], capture_output=True, text=True,
                                                    check=True).stdout.split())
    assert n > 100000 and zeros > 6000
    assert bad == 0
