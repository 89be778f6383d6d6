"""The verify kernel on the FP64 pipe (csrc/kernels_verify_fp.cu): its field,
point and digit arithmetic against exact integers on the host, its verdicts
against the oracle at the edges of its blocks and on signatures whose two sums
meet (equal or opposite points)."""
from __future__ import annotations

import ctypes
import glob
import os
import random
import subprocess

import numpy as np
import pytest

from conftest import N, NATIVE, P, ROOT, ecdsa_corpus, opaque_rows_corpus, schnorr_corpus

G = (0x79BE667EF9DCBBAC55A06295CE870B07029BFCDB2DCE28D959F2815B16F81798,
     0x483ADA7726A3C4655DA4FBFC0E1108A8FD17B448A68554199C47D08FFB10D4B8)
LAMBDA = 0x5363AD4CC05C30E0A5261C028812645A122E22EA20816678DF02967C1B23BD72
Digits = ctypes.c_double * 5
Limbs = ctypes.c_uint32 * 8


@pytest.fixture(scope="module")
def fp():
    so = os.path.join(NATIVE, "libfpfield_host.so")
    src = os.path.join(NATIVE, "fpfield_host.cpp")
    deps = [src] + glob.glob(os.path.join(ROOT, "ultrafastsecp256k1_b200", "csrc", "*.cuh"))
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        # the products round downwards: the compiler may not assume round-to-nearest
        subprocess.run(["g++", "-O2", "-std=c++17", "-frounding-math", "-fPIC", "-shared", "-o", so, src], check=True)
    return ctypes.CDLL(so)


def limbs(v):
    return Limbs(*[(v >> (32 * i)) & 0xFFFFFFFF for i in range(8)])


def value(d):
    return sum(int(x) << (52 * i) for i, x in enumerate(d))


def strict(rnd):
    """Strict digits, often at the ends of their range."""
    out = []
    for i in range(5):
        m = 2**51 if i < 4 else 2**47 + 4096
        out.append(rnd.choice([m, -m, m - 1, 1 - m, 0, 1, -1]) if rnd.random() < 0.4 else rnd.randint(-m, m))
    return out


def unsigned(rnd):
    """The digits of an unpacked 256-bit coordinate."""
    v = rnd.choice([0, 1, 2**256 - 1, P - 1]) if rnd.random() < 0.2 else rnd.randrange(2**256)
    return [(v >> (52 * i)) & (2**52 - 1) for i in range(5)]


def ec_add(a, b):
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


# op -> (value of a, b, x, y, operands: s strict, u strict or unsigned, d difference of two strict)
OPS = {0: (lambda a, b, x, y: a * b, "ub"), 1: (lambda a, b, x, y: a * a, "s"),
       2: (lambda a, b, x, y: a * b - x, "ub"), 3: (lambda a, b, x, y: 2 * a * a, "s"),
       4: (lambda a, b, x, y: 3 * a * a, "s"), 5: (lambda a, b, x, y: a * a - 2 * x, "s"),
       6: (lambda a, b, x, y: a * a - x - y, "s"), 7: (lambda a, b, x, y: a * a - x - 2 * y, "s"),
       8: (lambda a, b, x, y: a * b - x * y, "d"), 9: (lambda a, b, x, y: a * b - 2 * x * x, "d"),
       10: (lambda a, b, x, y: a, "u")}


@pytest.mark.parametrize("op", sorted(OPS))
def test_field_operations_are_exact(fp, op):
    """Every operation mod p, digits of the result within their strict bounds,
    its value in (-p, p) and its packed limbs canonical."""
    rnd = random.Random(op)
    want, form = OPS[op]
    for _ in range(3000):
        a, b, x, y = (strict(rnd) for _ in range(4))
        if form[0] == "u" and rnd.random() < 0.5:
            a = unsigned(rnd)
        elif form[0] == "d" or (form == "ub" and rnd.random() < 0.5):
            a = [p - q for p, q in zip(a, strict(rnd))]
        out = Digits()
        fp.fp_op(op, Digits(*a), Digits(*b), Digits(*x), Digits(*y), out)
        r = list(out)
        w = want(*map(value, (a, b, x, y)))
        assert all(float(int(v)) == v for v in r) and all(abs(v) <= 2**51 for v in r[:4])
        if op == 10:
            assert value(r) == w
            continue
        assert (value(r) - w) % P == 0 and abs(value(r)) < P and abs(r[4]) <= 2**47 + 4096
        packed = Limbs()
        fp.fp_pack(out, packed)
        assert sum(v << (32 * i) for i, v in enumerate(packed)) == w % P


def test_unpack_keeps_the_value(fp):
    rnd = random.Random(1)
    for v in [0, 1, P - 1, P, 2**256 - 1] + [rnd.randrange(2**256) for _ in range(500)]:
        out = Digits()
        fp.fp_unpack(limbs(v), out)
        assert value(out) == v and all(0 <= d < 2**52 for d in out)


def test_joint_digits_and_table(fp):
    """k P over the joint digits for scalars at the ends of their range, units and
    their neighbours, short digit strings, and random ones."""
    rnd = random.Random(2)
    special = [0, 1, 2, 3, 4, 5, 7, 8, 9, 63, 64, N - 1, N - 2, N // 2, N // 2 + 1, LAMBDA, N - LAMBDA,
               LAMBDA * LAMBDA % N, (1 + LAMBDA) % N, 8 * LAMBDA % N, (64 + 7 * LAMBDA) % N]
    for k in special + [rnd.randrange(N) for _ in range(60)]:
        pt = ec_mul(rnd.randrange(1, N), G)
        out = (ctypes.c_uint32 * 24)()
        finite = fp.fp_point_mul(limbs(k), limbs(pt[0]), limbs(pt[1]), out)
        expect = ec_mul(k, pt)
        assert bool(finite) == (expect is not None)
        if finite:
            X, Y, Z = (sum(out[8 * c + i] << (32 * i) for i in range(8)) for c in range(3))
            zi = pow(Z, -1, P)
            assert (X * zi * zi % P, Y * zi**3 % P) == expect


# ---- on the GPU -----------------------------------------------------------------

def _be(v):
    return np.frombuffer(v.to_bytes(32, "big"), np.uint8)


@pytest.fixture(scope="module")
def fp_ctx():
    """A context whose calls of every size take the FP64 kernel."""
    import ultrafastsecp256k1_b200 as uf
    with uf.GpuContext(0) as ctx:
        for k in (0, 1):
            ctx.set_small_variant(k, -1)
            ctx.set_lanes(k, 1)
            ctx.set_inversion_group(k, 128)
        yield ctx


def check_sizes(fp_ctx, oracle, n):
    import ultrafastsecp256k1_b200 as uf
    m = min(n, 701)
    order = np.random.default_rng(n).integers(0, m, n)
    em, ep, es = ecdsa_corpus(oracle, m, 17)
    sm, sp, ss = schnorr_corpus(oracle, m, 18, tamper=0.1)
    rows = opaque_rows_corpus(oracle, m, 19)
    assert (fp_ctx.ecdsa_verify_batch(em[order], ep[order], es[order]) ==
            oracle.ecdsa_verify_batch(em, ep, es)[order]).all()
    assert (fp_ctx.schnorr_verify_batch(sm[order], sp[order], ss[order]) ==
            oracle.schnorr_verify_batch(sm, sp, ss)[order]).all()
    L = uf.load_library()
    L.ufsecp_gpu_ecdsa_verify_opaque_rows.argtypes = [uf._vp, uf._vp, ctypes.c_size_t, ctypes.c_size_t, uf._vp]
    out = np.full(n, 9, np.uint8)
    tiled = np.ascontiguousarray(rows[order])
    assert L.ufsecp_gpu_ecdsa_verify_opaque_rows(fp_ctx.handle, tiled.ctypes.data, 129, n, out.ctypes.data) == 0
    assert (out == oracle.ecdsa_verify_opaque_rows(rows, 129)[order]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 147, 149, 4737, 18945, 37887, 37888, 37889, 80001])
def test_block_edges(fp_ctx, oracle, n):
    """One item to two rounds of full blocks, around the block and grid sizes
    (148 SMs, up to 256 items each), both schemes and the opaque rows."""
    check_sizes(fp_ctx, oracle, n)


def meeting_signatures(oracle):
    """ECDSA items whose generator and key sums are equal (valid signatures by
    construction: R = 2 u1 G) or opposite (R = infinity), and BIP-340 items with
    s G = e P (R = infinity) or s G = -e P."""
    rnd = random.Random(9)
    em, ep, es, sm, sp, ss = ([] for _ in range(6))
    while len(em) < 12:
        d, u1 = rnd.randrange(1, N), rnd.randrange(1, N)
        r = ec_mul(2 * u1 % N, G)[0] % N
        z = (r * d if len(em) % 2 == 0 else -r * d) % N
        s = z * pow(u1, -1, N) % N
        if s > N // 2:
            continue
        Q = ec_mul(d, G)
        em.append(_be(z))
        ep.append(np.concatenate([np.array([2 + (Q[1] & 1)], np.uint8), _be(Q[0])]))
        es.append(np.concatenate([_be(r), _be(s)]))
    import hashlib
    tag = hashlib.sha256(b"BIP0340/challenge").digest()
    for k in range(8):
        d = rnd.randrange(1, N)
        Q = ec_mul(d, G)
        d = d if Q[1] % 2 == 0 else N - d
        r, msg = rnd.randrange(P).to_bytes(32, "big"), rnd.randbytes(32)
        px = Q[0].to_bytes(32, "big")
        e = int.from_bytes(hashlib.sha256(tag + tag + r + px + msg).digest(), "big") % N
        s = (e * d if k % 2 == 0 else -e * d) % N
        sm.append(np.frombuffer(msg, np.uint8))
        sp.append(np.frombuffer(px, np.uint8))
        ss.append(np.concatenate([np.frombuffer(r, np.uint8), _be(s)]))
    return [np.stack(v) for v in (em, ep, es, sm, sp, ss)]


def test_meeting_signatures_are_what_they_say(oracle):
    em, ep, es, sm, sp, ss = meeting_signatures(oracle)
    assert oracle.ecdsa_verify_batch(em, ep, es).tolist() == [1, 0] * 6
    assert not oracle.schnorr_verify_batch(sm, sp, ss).any()


def check_meeting(fp_ctx, oracle):
    em, ep, es, sm, sp, ss = meeting_signatures(oracle)
    om, op, os_ = ecdsa_corpus(oracle, 60, 23)
    em, ep, es = (np.concatenate([a, b])[::-1].copy() for a, b in ((em, om), (ep, op), (es, os_)))
    assert (fp_ctx.ecdsa_verify_batch(em, ep, es) == oracle.ecdsa_verify_batch(em, ep, es)).all()
    om, op, os_ = schnorr_corpus(oracle, 60, 24, tamper=0.1)
    sm, sp, ss = (np.concatenate([a, b])[::-1].copy() for a, b in ((sm, om), (sp, op), (ss, os_)))
    assert (fp_ctx.schnorr_verify_batch(sm, sp, ss) == oracle.schnorr_verify_batch(sm, sp, ss)).all()


@pytest.mark.gpu
def test_sums_that_meet(fp_ctx, oracle):
    """Equal and opposite sums among ordinary items."""
    check_meeting(fp_ctx, oracle)


@pytest.fixture(scope="module")
def team_ctx():
    """A context whose calls of every size take the small-call kernel (four warps per 32 signatures)."""
    import ultrafastsecp256k1_b200 as uf
    with uf.GpuContext(0) as ctx:
        for k in (0, 1):
            ctx.set_lanes(k, 2, 1 << 22)
        yield ctx


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 147 * 32 + 5, 9473])
def test_team_block_edges(team_ctx, oracle, n):
    """Part of a block to more blocks than run at once."""
    check_sizes(team_ctx, oracle, n)


@pytest.mark.gpu
def test_team_sums_that_meet(team_ctx, oracle):
    check_meeting(team_ctx, oracle)


@pytest.fixture(scope="module")
def plain_ctx():
    import ultrafastsecp256k1_b200 as uf
    with uf.GpuContext(0) as ctx:
        yield ctx


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8191, 8192, 8193, 37889, 47360, 47361, 56832, 56833, 75809])
def test_chunks_and_last_waves(plain_ctx, oracle, n):
    """Host calls around the size from which staging is packed in pieces, and
    around whole waves (256 items on each of 148 SMs) plus the last waves that
    run in their own form: up to 64 items per SM, up to 128, and more."""
    check_sizes(plain_ctx, oracle, n)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [37889, 47361, 56832, 56833])
def test_device_last_waves(plain_ctx, oracle, n):
    import torch
    m, p, s = schnorr_corpus(oracle, 701, 18, tamper=0.1)
    order = np.random.default_rng(n).integers(0, 701, n)
    want = oracle.schnorr_verify_batch(m, p, s)[order]
    d = [torch.from_numpy(np.ascontiguousarray(a[order])).cuda() for a in (m, p, s)]
    out = torch.full((n + 1,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    plain_ctx.schnorr_verify_device(*(a.data_ptr() for a in d), n, out.data_ptr(), stream=stream.cuda_stream)
    stream.synchronize()
    got = out.cpu().numpy()
    assert (got[:n] == want).all() and got[n] == 7


@pytest.mark.gpu
def test_jobs_packed_in_pieces(plain_ctx, oracle):
    em, ep, es = ecdsa_corpus(oracle, 701, 17)
    sm, sp, ss = schnorr_corpus(oracle, 701, 18, tamper=0.1)
    rng = np.random.default_rng(5)
    jobs, want = [], []
    for k, n in ((1, 9001), (0, 1), (0, 5003), (1, 33), (1, 0), (0, 3000), (1, 4096), (0, 21000), (1, 2)):
        order = rng.integers(0, 701, n)
        src = (em, ep, es) if k == 0 else (sm, sp, ss)
        jobs.append((k, *(np.ascontiguousarray(a[order]) for a in src)))
        ref = oracle.ecdsa_verify_batch(em, ep, es) if k == 0 else oracle.schnorr_verify_batch(sm, sp, ss)
        want.append(ref[order])
    for got, ref in zip(plain_ctx.verify_jobs(jobs), want):
        assert (got == ref).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4736, 4737, 9471, 9472])
def test_two_warps_per_32_signatures(team_ctx, oracle, n):
    """Around a block per SM (four warps up to it, two above) and two."""
    check_sizes(team_ctx, oracle, n)


@pytest.mark.gpu
def test_two_warp_sums_that_meet(team_ctx, oracle):
    em, ep, es, sm, sp, ss = meeting_signatures(oracle)
    order = np.random.default_rng(3).integers(0, len(em), 4800)
    assert (team_ctx.ecdsa_verify_batch(em[order], ep[order], es[order]) ==
            oracle.ecdsa_verify_batch(em, ep, es)[order]).all()
    order = np.random.default_rng(4).integers(0, len(sm), 4800)
    assert not team_ctx.schnorr_verify_batch(sm[order], sp[order], ss[order]).any()
