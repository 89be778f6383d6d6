"""Digit ranges of the FP64 field (csrc/fd.cuh, jacd.cuh) at their ends: operands
whose top digit is as large as the others, sums and differences, the general point
addition where its terms lie near +-2^255."""
import ctypes
import glob
import os
import random
import subprocess

import pytest

from conftest import NATIVE, P, ROOT
from test_fp_verify import OPS, Digits, Limbs, fp, limbs, value  # noqa: F401


@pytest.fixture(scope="module")
def jd():
    so = os.path.join(NATIVE, "libjacd_host.so")
    src = os.path.join(NATIVE, "jacd_host.cpp")
    deps = [src] + glob.glob(os.path.join(ROOT, "ultrafastsecp256k1_b200", "csrc", "*.cuh"))
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-frounding-math", "-fPIC", "-shared", "-o", so, src], check=True)
    return ctypes.CDLL(so)


def wide(rnd, top=2**51):
    """Digits in [-2^51, 2^51], the top one too, often at the ends."""
    return [rnd.choice([m, -m, m - 1, 1 - m]) if rnd.random() < 0.5 else rnd.randint(-m, m)
            for m in (2**51, 2**51, 2**51, 2**51, top)]


@pytest.mark.parametrize("op", sorted(set(OPS) - {10}))
def test_operations_take_a_large_top_digit(fp, op):  # noqa: F811
    rnd = random.Random(100 + op)
    want, _ = OPS[op]
    for k in range(2000):
        top = 2**50 if k % 2 else 2**49      # the top products of a b - 2 x^2 together below 2^103
        a, b, x, y = (wide(rnd, top) for _ in range(4))
        out = Digits()
        fp.fp_op(op, Digits(*a), Digits(*b), Digits(*x), Digits(*y), out)
        r = list(out)
        assert (value(r) - want(*map(value, (a, b, x, y)))) % P == 0
        assert all(abs(v) <= 2**51 for v in r[:4]) and abs(value(r)) < P


def test_strict_of_any_top_digit(fp):  # noqa: F811
    rnd = random.Random(7)
    for _ in range(2000):
        a = [rnd.randint(-2**53 + 1, 2**53 - 1) for _ in range(4)] + [rnd.randint(-2**52, 2**52)]
        out = Digits()
        fp.fp_op(10, Digits(*a), Digits(*a), Digits(*a), Digits(*a), out)
        assert value(out) == value(a) and all(abs(v) <= 2**51 for v in list(out)[:4])


def test_sums_and_differences(jd):
    rnd = random.Random(8)
    for _ in range(2000):
        a, b = wide(rnd), wide(rnd)
        s, d = Digits(), Digits()
        jd.jd_add_sub(Digits(*a), Digits(*b), s, d)
        assert value(s) == value(a) + value(b) and value(d) == value(a) - value(b)
        assert all(abs(v) <= 2**51 for v in list(s)[:4] + list(d)[:4])


def test_general_addition_stays_in_range(jd):
    """U, r and H chosen so that V = U H^2 and r^2 - H^3 - V lie within 2^219 of
    -2^255 and 2^255: X = r^2 - H^3 - 2 V taken as a difference of two reduced
    values leaves (-p, p) there, and its packed limbs are then wrong."""
    rnd = random.Random(9)
    done = 0
    while done < 400:
        H = rnd.randrange(1, P)
        sign = rnd.choice([1, -1])
        V = (-sign * 2**255 + rnd.randint(-2**219, 2**219)) % P
        s = (sign * 2**255 + rnd.randint(-2**219, 2**219)) % P
        r2 = (s + H**3 + V) % P
        r = pow(r2, (P + 1) // 4, P)
        if r * r % P != r2:
            continue
        done += 1
        U, Y1 = V * pow(H * H, -1, P) % P, rnd.randrange(P)
        a = [U, Y1, 1]
        b = [(U + H) % P, (Y1 + r) % P, 1]
        digits, packed = (ctypes.c_double * 15)(), (ctypes.c_uint32 * 24)()
        jd.jd_add((ctypes.c_uint32 * 24)(*sum((list(limbs(v)) for v in a), [])),
                  (ctypes.c_uint32 * 24)(*sum((list(limbs(v)) for v in b), [])), digits, packed)
        X = (r * r - H**3 - 2 * V) % P
        want = [X, (r * (V - X) - Y1 * H**3) % P, H]
        for c in range(3):
            v = value(list(digits)[5 * c:5 * c + 5])
            assert abs(v) < P and (v - want[c]) % P == 0
            assert sum(w << (32 * i) for i, w in enumerate(packed[8 * c:8 * c + 8])) == want[c]


def test_squares(jd):
    rnd = random.Random(10)
    for v in [0, 1, 3, P - 1, 7] + [rnd.randrange(P) for _ in range(40)]:
        assert jd.jd_is_square(limbs(v)) == (v == 0 or pow(v, (P - 1) // 2, P) == 1)
