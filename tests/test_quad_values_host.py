"""The four values of a pair of factors (theboss_gb300/csrc/boss_quad.cuh) compiled for
the host and checked against exact integers: each within 2^-55 of its own size, also
where the factors cancel far below their largest sums."""
import os
import shutil
import subprocess
from fractions import Fraction as F

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LOW = [(1, 1), (-1, -1), (1, -1), (-1, 1)]  # the kernel's order


def test_values_keep_their_digits(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "quad_value_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", os.path.join(HERE, "native", "quad_value_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    seen = {0: 0, 1: 0, "zero": 0}
    for line in subprocess.run([exe, "5", "6000"], check=True, capture_output=True, text=True).stdout.splitlines():
        v = list(map(int, line.split()))
        nd, one, u = v[0], v[1], [v[18 + 5 * a:23 + 5 * a] for a in range(v[0])]
        for k, (d0, d1) in enumerate(LOW):
            re, im, l, small = v[2 + 4 * k:6 + 4 * k]
            s = [0, 0, one, 0]
            for a in range(nd):
                d = (d0, d1)[a] if a < 2 else u[a][0]
                for c in range(4):
                    s[c] += d * u[a][1 + c]
            exact = s[0] * s[2] - s[1] * s[3], s[0] * s[3] + s[1] * s[2]
            size = max(abs(exact[0]), abs(exact[1]))
            seen[small] += 1
            assert abs(re) <= 2 ** 62 and abs(im) <= 2 ** 62
            if size == 0:
                assert re == 0 and im == 0
                seen["zero"] += 1
                continue
            assert max(abs(re), abs(im)) >= 2 ** 61 - 1
            for c, got in enumerate((re, im)):
                # 16 roundings of the coefficients at most (half a unit of 2^48 each) over 2^108, truncations 2^-60
                assert abs(F(got) * F(2) ** (l + 35) - exact[c]) <= F(size) * F(2) ** -55, (nd, k, small, l)
    assert min(seen.values()) > 100
