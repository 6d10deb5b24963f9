"""Four codes per step over pairs of factors (theboss_gb300/csrc/boss_quad.cuh): the
arithmetic compiled for the host with nvcc and checked against exact integers: the
four sign combinations of the low digits, odd and even factor counts, small
factors, exact zeros and a dominating digit."""
import os
import shutil
import subprocess
from fractions import Fraction as F

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LOW = [(1, 1), (-1, -1), (1, -1), (-1, 1)]  # the kernel's order


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("quad") / "quad_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", os.path.join(HERE, "native", "quad_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = []
    for seed in (3, 8):
        out += subprocess.run([exe, str(seed), "450"], check=True, capture_output=True, text=True).stdout.splitlines()
    return out


def _mul(a, b):
    return a[0] * b[0] - a[1] * b[1], a[0] * b[1] + a[1] * b[0]


def test_quad_products(lines):
    zeros = 0
    for line in lines:
        v = list(map(int, line.split()))
        nf, nd, outer, e = v[:4]
        got = [(F(v[4 + 3 * k]) * F(2) ** (e + v[6 + 3 * k]), F(v[5 + 3 * k]) * F(2) ** (e + v[6 + 3 * k])) for k in range(4)]
        u = [(v[16 + 2 * i], v[17 + 2 * i]) for i in range(nd * nf)]
        exact, largest = [], []
        for d0, d1 in LOW:
            sg = [d0, d1] + [-1 if (outer >> (a - 2)) & 1 else 1 for a in range(2, nd)]
            p = (1, 0)
            for f in range(nf):
                p = _mul(p, (sum(sg[a] * u[a * nf + f][0] for a in range(nd)),
                             sum(sg[a] * u[a * nf + f][1] for a in range(nd))))
            exact.append(p)
        # every pair's coefficients are rounded to half a unit of 2^64 (nd of them, doubled by E's two signs,
        # and its truncated product, two units), every chain product is within 2 units of a value of 61 bits:
        # relative to the product of the factors' largest sums B_f (2^62 units each, 2^124 a pair)
        B = 1.0
        for f in range(nf):
            B *= float(sum(max(abs(u[a * nf + f][0]), abs(u[a * nf + f][1])) for a in range(nd))) * 2.0 ** 0.5 + 1.0
        bound = 0.0
        for f in range(0, nf - 1, 2):
            pair = 1.0
            for h in (f, f + 1):
                pair *= float(sum(max(abs(u[a * nf + h][0]), abs(u[a * nf + h][1])) for a in range(nd))) * 2.0 ** 0.5 + 1.0
            bound += (2.0 * nd + 4.0) * 2.0 ** 64 / pair  # units of 2^64 of the pair's largest product
        tol = B * (bound + nf * 2.0 ** -56)
        top = max(max(abs(x) for x in g) for g in got)
        for k in range(4):
            for c in range(2):
                err = abs(got[k][c] - exact[k][c])
                assert err <= F(tol) + top * F(2) ** -58, (nf, nd, outer, k, float(err), tol)
            if exact[k] == (0, 0) and all(x == 0 for g in got for x in g):
                zeros += 1
    assert zeros > 0


def test_quad_accuracy_on_full_size_factors(lines):
    """Factors that use their bits: products within 2^-54 of their typical size."""
    worst = 0.0
    for line in lines:
        v = list(map(int, line.split()))
        nf, nd, outer, e = v[:4]
        u = [(v[16 + 2 * i], v[17 + 2 * i]) for i in range(nd * nf)]
        if min(max(abs(x) for x in w) for w in u) < 2 ** 54:
            continue
        sums = []
        for d0, d1 in LOW:
            sg = [d0, d1] + [-1 if (outer >> (a - 2)) & 1 else 1 for a in range(2, nd)]
            sums.append([(sum(sg[a] * u[a * nf + f][0] for a in range(nd)),
                          sum(sg[a] * u[a * nf + f][1] for a in range(nd))) for f in range(nf)])
        ex = []
        for s in sums:
            p = (1, 0)
            for z in s:
                p = _mul(p, z)
            ex.append(p)
        size = max(max(abs(x) for x in p) for p in ex)
        for k in range(4):
            for c in range(2):
                worst = max(worst, float(abs(F(v[4 + 3 * k + c]) * F(2) ** (e + v[6 + 3 * k]) - ex[k][c]) / size))
    assert 0.0 < worst < 2.0 ** -50, worst  # small sums inside a pair amplify its 2^64 unit
