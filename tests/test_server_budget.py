"""A server's memory budget and its key table (csrc/server_budget.h): budgets that
held one launch slot and a table of 576-byte slots are taken with 768-byte ones."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import NATIVE, ROOT, _newer, schnorr_corpus

OLD, NEW, LAUNCH = 576, 768, 36 << 20


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(NATIVE, "libserver_budget_host.so")
    src = os.path.join(NATIVE, "server_budget_host.cpp")
    if not _newer(so, src, os.path.join(ROOT, "ultrafastsecp256k1_b200", "csrc", "server_budget.h")):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so, src], check=True)
    lib = ctypes.CDLL(so)
    lib.sb_fit.argtypes = [ctypes.c_uint32, ctypes.c_uint32] + [ctypes.c_uint64] * 3
    return lib


@pytest.mark.parametrize("log2", [0, 8, 9, 18, 24])
def test_table_fits_or_is_halved(lib, log2):
    def fit(budget):
        return lib.sb_fit(log2, 8, NEW, budget, LAUNCH)
    old, new = ((s << log2) + 256 if log2 else 0 for s in (OLD, NEW))
    half = log2 - 1 if log2 > 8 else 0
    assert fit(0) == fit(LAUNCH - 1) == fit(LAUNCH + old - 1) == -1
    assert fit(LAUNCH + new) == fit(8 << 40) == log2
    if log2:
        assert fit(LAUNCH + old) == fit(LAUNCH + new - 1) == half
        assert (NEW << half if half else 0) + 256 <= old


@pytest.mark.gpu
def test_server_between_the_two_sizes(oracle):
    import ultrafastsecp256k1_b200 as uf
    m, p, s = schnorr_corpus(oracle, 300, 71, tamper=0.1)
    want = oracle.schnorr_verify_batch(m, p, s)
    with uf.GpuContext(0) as ctx:
        with uf.Server(ctx, slots=1, key_cache_log2=0) as srv:
            slot = srv.stats()["reserved_bytes"]
        for extra, made in (((OLD << 18) + 256, NEW << 17), ((NEW << 18) + 256, NEW << 18)):
            with uf.Server(ctx, slots=2, key_cache_log2=18, memory_budget_bytes=slot + extra) as srv:
                assert srv.stats()["reserved_bytes"] >= slot + made
                assert srv.stats()["reserved_bytes"] <= slot + extra
                for _ in range(2):
                    assert (srv.wait(srv.submit([(1, m, p, s)]))[0] == want).all()
        with pytest.raises(uf.UfsecpError):
            uf.Server(ctx, slots=2, key_cache_log2=18, memory_budget_bytes=slot + (OLD << 18) + 255)
