"""A host-buffer call whose staging exists allocates nothing on the host, so that no
std::bad_alloc can end it while copies of its chunks are still in flight."""
import os
import subprocess
import sys

import pytest

from conftest import NATIVE, ROOT, _newer

SCRIPT = """
import ctypes, sys
import numpy as np
import ultrafastsecp256k1_b200 as uf
lib = ctypes.CDLL(sys.argv[1])
rng = np.random.default_rng(1)
n = 100000
m, p, s = (rng.integers(0, 256, (n, w), dtype=np.uint8) for w in (32, 32, 64))
out = np.zeros(n, np.uint8)
with uf.GpuContext(0) as ctx:
    fn = uf.load_library().ufsecp_gpu_schnorr_verify_batch
    for size in (n, 100, 9000, n):
        for armed in (False, True):
            if armed:
                lib.cn_arm()
            rc = fn(ctx.handle, m.ctypes.data, p.ctypes.data, s.ctypes.data, size, out.ctypes.data)
            count = lib.cn_disarm()
            assert rc == 0
        print(size, count)
"""


@pytest.mark.gpu
def test_repeated_host_calls_allocate_nothing():
    so = os.path.join(NATIVE, "libcount_new.so")
    src = os.path.join(NATIVE, "count_new.cpp")
    if not _newer(so, src):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so, src], check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT, so], cwd=ROOT, env={**os.environ, "LD_PRELOAD": so},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split("\n")[:-1] == ["100000 0", "100 0", "9000 0", "100000 0"]
