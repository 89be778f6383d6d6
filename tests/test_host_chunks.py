"""How a host-buffer call is cut into chunks (csrc/host_chunks.h): whole waves for
the FP64 kernel, doubling chunks for the integer kernels."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import NATIVE, ROOT, _newer, schnorr_corpus

WAVE = 148 * 256
WAIT = 1 << 40


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(NATIVE, "libhost_chunks_host.so")
    src = os.path.join(NATIVE, "host_chunks_host.cpp")
    if not _newer(so, src, os.path.join(ROOT, "ultrafastsecp256k1_b200", "csrc", "host_chunks.h")):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so, src], check=True)
    lib = ctypes.CDLL(so)
    lib.hc_cut.argtypes = [ctypes.c_size_t, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_int]
    lib.hc_count.argtypes = [ctypes.c_size_t, ctypes.c_size_t, ctypes.c_int]
    return lib


def cut(lib, wave, items):
    out = np.zeros(64, np.uint64)
    return [int(v) for v in out[:lib.hc_cut(wave, items, out.ctypes.data, 64)]]


def test_waves(lib):
    assert cut(lib, WAVE, 1) == [1]
    assert cut(lib, WAVE, WAVE) == [WAVE]
    assert cut(lib, WAVE, WAVE + 1) == [WAVE, 1 | WAIT]
    assert cut(lib, WAVE, 3 * WAVE // 2) == [WAVE, WAVE // 2 | WAIT]
    assert cut(lib, WAVE, 3 * WAVE // 2 + 1) == [WAVE, WAVE // 2 + 1]


def test_doubling_chunks_of_the_integer_kernels(lib):
    """No chunk waits, and a call just above a wave is not cut into a wave and a rest."""
    assert cut(lib, 0, 16384) == [16384]
    assert cut(lib, 0, WAVE + 1) == [16384, WAVE + 1 - 16384]
    assert cut(lib, 0, 131073) == [16384, 32768, 65536, 131073 - 114688]
    assert cut(lib, 0, 400000) == [16384, 32768, 65536, 131072, 131072, 400000 - 376832]


@pytest.mark.parametrize("wave", [0, WAVE, 256])
def test_every_item_once(lib, wave):
    for items in (0, 1, 255, 257, 16385, WAVE + 1, 200000, 262145):
        if items > 60 * (wave or 1 << 20):
            continue
        sizes = [v & ~WAIT for v in cut(lib, wave, items)]
        assert sum(sizes) == items and all(sizes)
        assert lib.hc_count(wave, items, 3) == min(3, len(sizes))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16384, 16385, 37889, 131073])
@pytest.mark.parametrize("small", [False, True])
def test_integer_kernels_host_calls(oracle, n, small):
    import ultrafastsecp256k1_b200 as uf
    m, p, s = schnorr_corpus(oracle, 701, 18, tamper=0.1)
    order = np.random.default_rng(n).integers(0, 701, n)
    with uf.GpuContext(0) as ctx:
        ctx.set_variant(1, 4)
        if small:
            ctx.set_small_variant(1, 6, 32768)
        got = ctx.schnorr_verify_batch(m[order], p[order], s[order])
        got2 = ctx.schnorr_verify_batch(m[order][:900], p[order][:900], s[order][:900])
    want = oracle.schnorr_verify_batch(m, p, s)[order]
    assert (got == want).all() and (got2 == want[:900]).all()
