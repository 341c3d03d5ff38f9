"""The certificate of the mixed SVD's finishing check (csrc/gram_bound.cuh): the bound of a cosine
from a Gram matrix with errors, and the error of an entry that it is told.

* The digits of fp64tc.cu in whole numbers: a row's element is round(x 2^(64 - e)) cut into eight
  signed base-256 digits, and the products of weight 8 and above are left out. What is left out per
  element, in units of 2^(e_a + e_b), is compared with the constant, over elements that make all of
  it as large as it can be and random ones.
* The bound against the exact cosine (in fractions) where every computed real sum is off by the
  whole error, in the direction that hides the cosine most."""
import os
import random
import subprocess
from fractions import Fraction

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("gram") / "gram_host")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "gram_host.cpp"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def bounds(exe, rows):
    text = "".join("%s %s %s %s %d\n" % (a.hex(), hi.hex(), hj.hex(), hb.hex(), c) for a, hi, hj, hb, c in rows)
    r = subprocess.run([exe], input=text, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    v = [float.fromhex(x) for x in r.stdout.split()]
    return v[0], v[1:]


def digits(q):
    d = [0] * 8
    for i in range(7, 0, -1):
        d[i] = ((q + 128) & 255) - 128
        q = (q - d[i]) >> 8
    d[0] = q
    assert abs(q) <= 128
    return d


def left_out(x, y):
    """|x y - the products of weight below 8|, x and y fractions below 1/2 in magnitude."""
    def cut(v):
        s = 1 if v >= 0 else -1
        return s * int(abs(v) * 2 ** 64 + Fraction(1, 2))
    a, b = digits(cut(x)), digits(cut(y))
    kept = sum(a[s] * b[t] * Fraction(1, 256 ** (s + t + 2)) for s in range(8) for t in range(8 - s))
    return abs(x * y - kept)


def test_omitted_products(exe):
    limit = Fraction(bounds(exe, [])[0])
    rng = random.Random(1)
    full = Fraction(sum(-128 * 256 ** (7 - i) for i in range(1, 8)) - 127 * 256 ** 7, 2 ** 64)
    half = Fraction(1, 2 ** 65)
    worst = Fraction(0)
    for x in (full, -full, full - half * Fraction(99, 100), -full + half * Fraction(99, 100)):
        for y in (full, -full, full - half * Fraction(99, 100)):
            worst = max(worst, left_out(x, y))
    assert worst > limit / 2  # (the constant is not far above what can happen)
    for _ in range(3000):
        v = []
        for _ in range(2):
            q = sum(rng.choice([-128, 127, rng.randrange(-128, 128)]) * 256 ** (7 - i) for i in range(8))
            q = max(-2 ** 63 + 1, min(2 ** 63 - 1, q))
            v.append(Fraction(q, 2 ** 64) * Fraction(2 ** 53 - 1, 2 ** 53))
        worst = max(worst, left_out(*v))
    assert worst <= limit


@pytest.mark.parametrize("cplx", [0, 1])
@pytest.mark.parametrize("k", [256, 8192, 1 << 20])
def test_bound_holds(exe, cplx, k):
    hb = Fraction(bounds(exe, [])[0]) * k
    rng = random.Random(k + cplx)
    rows, true = [], []
    for _ in range(2000):
        hii, hjj = (Fraction(rng.choice([0.0625, 0.0625 * (1 + rng.random()), rng.uniform(0.0625, k / 4)])) for _ in range(2))
        ang = rng.choice([0.0, 1.0, rng.random()])
        c = Fraction(10.0 ** rng.uniform(-17, -12))
        # h_ij = c (cos, sin) up to their own rounding: taken as they are
        re, im = c * Fraction((1 - ang * ang / 2)), (c * Fraction(ang) if cplx else Fraction(0))
        true.append((re * re + im * im) / (hii * hjj))
        cre, cim = max(re - hb, Fraction(0)), max(im - hb, Fraction(0))
        a = float((cre * cre + cim * cim)) ** 0.5
        rows.append((a, float(hii + hb), float(hjj + hb), float(hb) * (1 + 2.0 ** -50), cplx))
    for b, t in zip(bounds(exe, rows)[1], true):
        assert Fraction(b) ** 2 >= t
