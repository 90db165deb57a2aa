"""Index of a replica chip (csrc/chip_index.h): inside the sequence for every
double, and the exact remainder wherever 64 bits hold the chip number."""
import os
import struct
import subprocess

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include "chip_index.h"
int main() {
  double k;
  int L;
  while (std::fread(&k, 8, 1, stdin) == 1 && std::fread(&L, 4, 1, stdin) == 1) std::printf("%d\n", tga::chip_index(k, L));
}
"""


def test_every_double_has_a_place(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "tart-gnss_b200", "csrc"), "-o", exe,
                           str(tmp_path / "t.cpp")])
    rng = np.random.default_rng(1)
    ks = [0.0, -0.0, 2.0 ** 52, 2.0 ** 52 - 1, 2.0 ** 62, 2.0 ** 63, -2.0 ** 63, 1e18, 1e19, -1e19, 1e20, 1e300, -1e300,
          float("inf"), float("-inf"), float("nan"), 2147483648.0, -2147483649.0]
    ks += list(np.floor(rng.uniform(-1, 1, 2000) * 2.0 ** rng.uniform(0, 66, 2000)))
    ks += [m * L + e for L in (1023, 4092, 10230, 20460) for m in (1, -1, 12345678901, -98765432101) for e in (-1, 0, 1)]
    cases = [(float(k), L) for k in ks for L in (1023, 2046, 8184, 20460)]
    data = b"".join(struct.pack("<di", k, L) for k, L in cases)
    got = [int(v) for v in subprocess.run([exe], input=data, stdout=subprocess.PIPE, check=True).stdout.split()]
    assert len(got) == len(cases)
    for (k, L), g in zip(cases, got):
        assert 0 <= g < L, (k, L, g)
        if abs(k) < 2.0 ** 63:
            assert g == int(k) % L, (k, L, g)
