"""Items that only a crafted input reaches: an ECDSA r that may stand for r + n,
sums that meet or cancel, a digest of zero, keys off the curve whose points have a
small order.  The check of csrc/isocheck.cuh against exact integers on the host,
the verdicts of every kernel form against the oracle, and that such items cost
about what ordinary ones do."""
from __future__ import annotations

import ctypes
import glob
import hashlib
import os
import random
import subprocess

import numpy as np
import pytest

from conftest import N, NATIVE, P, ROOT, ecdsa_corpus, schnorr_corpus

G = (0x79BE667EF9DCBBAC55A06295CE870B07029BFCDB2DCE28D959F2815B16F81798,
     0x483ADA7726A3C4655DA4FBFC0E1108A8FD17B448A68554199C47D08FFB10D4B8)
Limbs = ctypes.c_uint32 * 8
NO, SOLVE, ON_CURVE, KEY_INF, PLAIN = range(5)
HOLDS = 256
SMALL_ORDERS = (3, 13, 3319)       # of points on the curve's quadratic twist


def limbs(v):
    return Limbs(*[(v >> (32 * i)) & 0xFFFFFFFF for i in range(8)])


def ec_add(a, b):
    """On y^2 = x^3 + k for any k: the formulas do not use it."""
    if a is None or b is None:
        return b if a is None else a
    if a[0] == b[0]:
        if (a[1] + b[1]) % P == 0:
            return None
        m = 3 * a[0] * a[0] * pow(2 * a[1], -1, P)
    else:
        m = (b[1] - a[1]) * pow(b[0] - a[0], -1, P)
    x = (m * m - a[0] - b[0]) % P
    return x, (m * (a[0] - x) - a[1]) % P


def ec_mul(k, pt):
    r = None
    while k:
        if k & 1:
            r = ec_add(r, pt)
        pt = ec_add(pt, pt)
        k >>= 1
    return r


def neg(pt):
    return pt and (pt[0], -pt[1] % P)


def lift(x, odd=0):
    y = pow((x**3 + 7) % P, (P + 1) // 4, P)
    if y * y % P != (x**3 + 7) % P:
        return None
    return x, (y if y % 2 == odd else P - y)


def point_from(x):
    """The point of the first x on the curve from x upwards."""
    while lift(x) is None:
        x += 1
    return lift(x)


def off_curve(rnd):
    while True:
        x = rnd.randrange(P)
        if lift(x) is None:
            return x


def twist_key(order, rnd):
    """x of a key off the curve: a point of that order on y^2 = x^3 + 7 c^3, c = x^3 + 7."""
    m = 2 * P + 2 - N
    assert m % order == 0
    while m % order == 0:
        m //= order
    while True:
        x = off_curve(rnd)
        c = (x**3 + 7) % P
        q = ec_mul(m, (x * c % P, c * c % P))
        while q is not None and ec_mul(order, q) is not None:
            q = ec_mul(order, q)
        if q is not None:
            return q[0] * pow(c, -1, P) % P


@pytest.fixture(scope="module")
def iso():
    so = os.path.join(NATIVE, "libisocheck_host.so")
    src = os.path.join(NATIVE, "isocheck_host.cpp")
    deps = [src] + glob.glob(os.path.join(ROOT, "ultrafastsecp256k1_b200", "csrc", "*.cuh"))
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-frounding-math", "-fPIC", "-shared", "-o", so, src], check=True)
    return ctypes.CDLL(so)


def check(iso, rnd, schnorr, key, b, B, r):
    """iso_check for the key (x, parity) and the generator's sum B, in both forms
    of the key's table where it is on the curve; the verdicts that the integers give."""
    x, odd = key
    z = rnd.randrange(1, P)
    jac = (0, 1, 0) if B is None else (B[0] * z * z % P, B[1] * z**3 % P, z)
    bj = (ctypes.c_uint32 * 24)(*sum((list(limbs(v)) for v in jac), []))
    pt = lift(x, odd)
    R = ec_add(ec_mul(b, pt), B) if pt else None
    want = R is not None and (R[0] == r or (not schnorr and r < P - N and R[0] == r + N))
    want = want and not (schnorr and R[1] % 2)
    got = []
    for unit in (0, 1):
        if unit and pt is None:
            continue
        res = iso.iso_check(schnorr, unit, limbs(x), limbs(pt[1] if pt else 0), odd, limbs(b), bj, limbs(r))
        st = res & 255
        if st not in (PLAIN, KEY_INF):
            assert (res & HOLDS != 0) == want, (schnorr, unit, st)
        got.append(st)
    return got


def key_of(pt):
    return pt[0], pt[1] & 1


def solve_for_key(R, B, b):
    """The key with b P + B = R."""
    return ec_mul(pow(b, -1, N), ec_add(R, neg(B)))


@pytest.mark.parametrize("schnorr", [0, 1])
def test_check_of_ordinary_items(iso, schnorr):
    rnd = random.Random(31 + schnorr)
    for k in range(24):
        b, B = rnd.randrange(1, N), ec_mul(rnd.randrange(1, N), G)
        R = ec_mul(rnd.randrange(1, N), G)
        Q = solve_for_key(R, B, b)
        r = R[0] if k % 3 else rnd.randrange(1, N)
        for odd in (0, 1):
            assert set(check(iso, rnd, schnorr, (Q[0], odd), b, B, r)) == {SOLVE}
        assert check(iso, rnd, schnorr, (off_curve(rnd), k & 1), b, B, r) == [SOLVE]


def test_check_of_r_plus_n(iso):
    """x(R) = r + n, x(R) = r below p - n, neither, and r at the ends of the range."""
    rnd = random.Random(33)
    for k in range(24):
        b, B = rnd.randrange(1, N), ec_mul(rnd.randrange(1, N), G)
        small = rnd.randrange(1, P - N - 2**64)
        R = point_from(small + (N if k % 2 else 0))
        Q = solve_for_key(R, B, b)
        r = R[0] % N
        for odd in (0, 1):
            assert set(check(iso, rnd, 0, (Q[0], odd), b, B, r)) == {SOLVE}
        check(iso, rnd, 0, key_of(Q), b, B, rnd.randrange(1, 2**128))
        check(iso, rnd, 0, (off_curve(rnd), 0), b, B, r)
        for end in (1, P - N - 1, P - N):
            check(iso, rnd, 0, key_of(Q), b, B, end)
        # BIP-340 has no second x
        check(iso, rnd, 1, key_of(Q), b, B, r)


@pytest.mark.parametrize("schnorr", [0, 1])
def test_check_of_meeting_sums(iso, schnorr):
    """A = B and A = -B, the wanted x met, met as r + n (ECDSA) and missed."""
    rnd = random.Random(35 + schnorr)
    for k in range(16):
        b = rnd.randrange(1, N)
        R = point_from(N + rnd.randrange(P - N - 2**64)) if k % 2 else ec_mul(rnd.randrange(1, N), G)
        B = ec_mul((N + 1) // 2, R)
        for Q in (ec_mul(pow(b, -1, N), B), neg(ec_mul(pow(b, -1, N), B))):
            for r in (R[0] % (P if schnorr else N), rnd.randrange(1, N), rnd.randrange(1, 2**128)):
                for odd in (0, 1):
                    assert set(check(iso, rnd, schnorr, (Q[0], odd), b, B, r)) <= {NO, SOLVE}


def test_check_without_a_generator_sum(iso):
    """ECDSA of a zero digest: R = b P."""
    rnd = random.Random(37)
    for k in range(12):
        b = rnd.randrange(1, N)
        R = point_from(N + rnd.randrange(P - N - 2**64)) if k % 2 else ec_mul(rnd.randrange(1, N), G)
        Q = ec_mul(pow(b, -1, N), R)
        assert set(check(iso, rnd, 0, key_of(Q), b, None, R[0] % N)) == {ON_CURVE}
        assert set(check(iso, rnd, 0, key_of(Q), b, None, rnd.randrange(1, N))) == {NO}
        # off the curve, the x of b P on the twist met (no second GLV half, whose
        # factor differs there): valid but for the key
        x, b = off_curve(rnd), rnd.randrange(1, 2**64)
        c = (x**3 + 7) % P
        X = ec_mul(b, (x * c % P, c * c % P))[0] * pow(c, -1, P) % P
        if X < N:
            assert check(iso, rnd, 0, (x, 0), b, None, X) == [ON_CURVE]


@pytest.mark.parametrize("schnorr", [0, 1])
def test_check_of_small_order_keys(iso, schnorr):
    """The table's path or the key's sum degenerates only off the curve, and then
    no item is left to the plain verification."""
    rnd = random.Random(39 + schnorr)
    for order in SMALL_ORDERS:
        for k in range(6):
            x, b = twist_key(order, rnd), rnd.randrange(1, N)
            for mult in (b, b - b % order or order):
                B = ec_mul(rnd.randrange(1, N), G)
                assert set(check(iso, rnd, schnorr, (x, k & 1), mult, B, rnd.randrange(1, N))) <= {NO, SOLVE, KEY_INF}
    B = ec_mul(5, G)
    if schnorr:
        assert set(check(iso, rnd, 1, key_of(ec_mul(7, G)), 0, B, B[0])) == {KEY_INF}


# ---- on the GPU -----------------------------------------------------------------

def _be(v):
    return np.frombuffer(v.to_bytes(32, "big"), np.uint8)


TAG = hashlib.sha256(b"BIP0340/challenge").digest()


def ecdsa_items(name, count, rnd):
    out = []
    while len(out) < count:
        d, z = rnd.randrange(1, N), rnd.randrange(N)
        Q, odd_key = ec_mul(d, G), None
        r, s = rnd.randrange(1, 2**128), rnd.randrange(1, N // 2)
        if name == "r_plus_n":
            R = point_from(N + rnd.randrange(P - N - 2**64))
            r = R[0] - N
            Q = ec_mul(pow(r, -1, N) * s % N, ec_add(R, neg(ec_mul(z * pow(s, -1, N) % N, G))))
        elif name in ("meet", "opposite"):
            u1 = rnd.randrange(1, N)
            r = ec_mul(2 * u1 % N, G)[0] % N
            z = (r * d if name == "meet" else -r * d) % N
            s = z * pow(u1, -1, N) % N
            if s > N // 2:
                continue
        elif name == "zero_digest":
            k = rnd.randrange(1, N)
            z, r = 0, ec_mul(k, G)[0] % N
            s = r * d * pow(k, -1, N) % N
            s = min(s, N - s)
            if len(out) % 3 == 2:
                r = r * 2 % N
        elif name == "small_order":
            odd_key = twist_key(SMALL_ORDERS[len(out) % 3], rnd)
            r = rnd.randrange(1, N)
        else:
            assert name == "small_r"
        x, par = (odd_key, 0) if odd_key else (Q[0], Q[1] & 1)
        out.append((_be(z), np.concatenate([np.array([2 + par], np.uint8), _be(x)]), np.concatenate([_be(r), _be(s)])))
    return [np.stack(v) for v in zip(*out)]


def schnorr_items(name, count, rnd):
    out = []
    for _ in range(count):
        d = rnd.randrange(1, N)
        Q = ec_mul(d, G)
        d = d if Q[1] % 2 == 0 else N - d
        x = Q[0] if name != "small_order" else twist_key(SMALL_ORDERS[len(out) % 3], rnd)
        r, msg = _be(rnd.randrange(P)), rnd.randbytes(32)
        e = int.from_bytes(hashlib.sha256(TAG + TAG + r.tobytes() + x.to_bytes(32, "big") + msg).digest(), "big") % N
        s = {"cancel": e * d % N, "meet": -e * d % N, "small_order": rnd.randrange(1, N)}[name]
        out.append((np.frombuffer(msg, np.uint8), _be(x), np.concatenate([r, _be(s)])))
    return [np.stack(v) for v in zip(*out)]


KINDS = [(0, k) for k in ("small_r", "r_plus_n", "meet", "opposite", "zero_digest", "small_order")] + \
        [(1, k) for k in ("cancel", "meet", "small_order")]


def crafted(kind, name, count=12):
    rnd = random.Random(f"{kind} {name}")
    return (ecdsa_items if kind == 0 else schnorr_items)(name, count, rnd)


def test_crafted_items_are_what_they_say(oracle):
    for name, want in (("r_plus_n", [1] * 12), ("meet", [1] * 12), ("opposite", [0] * 12),
                       ("zero_digest", [1, 1, 0] * 4), ("small_order", [0] * 12), ("small_r", [0] * 12)):
        assert oracle.ecdsa_verify_batch(*crafted(0, name)).tolist() == want, name
    for name in ("cancel", "meet", "small_order"):
        assert not oracle.schnorr_verify_batch(*crafted(1, name)).any()


def corpus(oracle, kind, seed):
    """Crafted items of every sort of this kind among 120 ordinary ones, and the oracle's verdicts."""
    parts = [crafted(kind, name) for k, name in KINDS if k == kind]
    parts.append(ecdsa_corpus(oracle, 120, seed) if kind == 0 else schnorr_corpus(oracle, 120, seed, tamper=0.1))
    rows = [np.concatenate(v) for v in zip(*parts)]
    return rows, (oracle.ecdsa_verify_batch if kind == 0 else oracle.schnorr_verify_batch)(*rows)


@pytest.mark.gpu
@pytest.mark.parametrize("form,n", [("threads", 700), ("threads", 40000), ("four warps", 700), ("two warps", 5000)])
def test_crafted_items_match_oracle(oracle, form, n):
    import ultrafastsecp256k1_b200 as uf
    with uf.GpuContext(0) as ctx:
        for k in (0, 1):
            ctx.set_lanes(k, *((1,) if form == "threads" else (2, 1 << 20)))
        for kind in (0, 1):
            rows, want = corpus(oracle, kind, 41)
            order = np.random.default_rng(n).integers(0, len(want), n)
            m, p, s = (a[order] for a in rows)
            call = ctx.ecdsa_verify_batch if kind == 0 else ctx.schnorr_verify_batch
            assert (call(m, p, s) == want[order]).all()


@pytest.mark.gpu
def test_crafted_items_in_jobs(oracle):
    """The same in mixed jobs: keys from the table (second call) and without one."""
    import ultrafastsecp256k1_b200 as uf
    with uf.GpuContext(0) as ctx:
        for k in (0, 1):
            ctx.set_lanes(k, 1)
        jobs, want = [], []
        for kind in (0, 1):
            rows, w = corpus(oracle, kind, 43)
            order = np.random.default_rng(kind).integers(0, len(w), 1500)
            jobs.append((kind, *(np.ascontiguousarray(a[order]) for a in rows)))
            want.append(w[order])
        for log2 in (12, 12, 0):
            if log2 == 0:
                ctx.set_key_table(0)
            for got, ref in zip(ctx.verify_jobs(jobs), want):
                assert (got == ref).all()


@pytest.mark.gpu
@pytest.mark.parametrize("kind,name", KINDS)
def test_crafted_items_cost_no_second_verification(kind, name):
    """One crafted item in a hundred among six waves on the device: at most half as
    much time again as ordinary items.  (Verified again by a lone lane behind its
    block, one such item in 256 takes longer than the block.)"""
    import torch

    import ultrafastsecp256k1_b200 as uf
    n = 148 * 256 * 6
    rng = np.random.default_rng(7)
    with uf.GpuContext(0) as ctx:
        def dev(a):
            return torch.from_numpy(np.ascontiguousarray(a)).cuda()
        msgs = rng.integers(0, 256, (n, 32), dtype=np.uint8)
        keys = rng.integers(1, 255, (n, 32), dtype=np.uint8)
        d_m, d_k = dev(msgs), dev(keys)
        d_p = torch.empty(n * (33 if kind == 0 else 32), dtype=torch.uint8, device="cuda")
        d_s = torch.empty(n * 64, dtype=torch.uint8, device="cuda")
        d_o = torch.empty(n, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ctx.sign_device(kind, d_m.data_ptr(), d_k.data_ptr(), d_m.data_ptr(), n, d_p.data_ptr(), d_s.data_ptr(),
                        d_o.data_ptr())
        torch.cuda.synchronize()
        rows = [msgs, d_p.cpu().numpy().reshape(n, -1), d_s.cpu().numpy().reshape(n, 64)]
        call = ctx.ecdsa_verify_device if kind == 0 else ctx.schnorr_verify_device
        items = crafted(kind, name)
        at = rng.choice(n, n // 100, replace=False)
        spoilt = [a.copy() for a in rows]
        for a, b in zip(spoilt, items):
            a[at] = b[np.arange(len(at)) % len(b)]
        times = []
        for side in (rows, spoilt):
            d, stream = [dev(a) for a in side], torch.cuda.Stream()
            best = float("inf")
            for _ in range(6):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                torch.cuda.synchronize()
                a.record(stream)
                call(*(x.data_ptr() for x in d), n, d_o.data_ptr(), stream=stream.cuda_stream)
                b.record(stream)
                torch.cuda.synchronize()
                best = min(best, a.elapsed_time(b))
            times.append(best)
    assert times[1] <= 1.5 * times[0], times
