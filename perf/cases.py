"""Timed workloads of the verify library: what a program that links it calls,
through the Python mirror of the C ABI, over the range of sizes it meets.

Every case is a plain dict; `prepare` builds its inputs (signed on the GPU from
the seed), `run` makes one pass and returns every verdict byte.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import ultrafastsecp256k1_b200 as uf

# Largest call of the device and host paths: the 2^20-signature batch of the
# library's own benchmark.
_MAX_ITEMS = 1 << 20
# Distinct keys behind the items of the job and serving cases (a node sees the
# same keys again and again; the draw over them is Zipf-like).
_KEY_POOL = 4096
# 32 x 32-bit multiply-adds of one per-signature verification: about 2000 field
# multiplications of 64 limb products; of one signature inside a random linear
# combination: two square roots and its share of the sums, about 800.
_VERIFY_MACS = 2000 * 64
_RLC_MACS = 800 * 64


def listed():
    return [
        # one signature per call: a wallet or a mempool checking transactions as they come
        {"name": "ecdsa_host_1", "path": "host", "scheme": "ecdsa", "n": 1, "calls": 16},
        # the Taproot key spends of a small block, host buffers
        {"name": "bip340_host_173", "path": "host", "scheme": "bip340", "n": 173, "calls": 1},
        # the benchmark's small ECDSA batch, already on the device
        {"name": "ecdsa_device_4096", "path": "device", "scheme": "ecdsa", "n": 4096},
        # a block's ECDSA inputs as the consensus code holds them (129-byte rows, libsecp's own layout)
        {"name": "ecdsa_rows_6011", "path": "rows", "scheme": "ecdsa", "n": 6011},
        # several blocks at once, host buffers (initial block download)
        {"name": "ecdsa_host_20011", "path": "host", "scheme": "ecdsa", "n": 20011, "calls": 1},
        # a device-side producer's medium batch, ragged size
        {"name": "bip340_device_50021", "path": "device", "scheme": "bip340", "n": 50021},
        # many callers' small batches in one call, both schemes, keys met before
        {"name": "jobs_400", "path": "jobs", "jobs": 400, "most": 4096},
        # a burst of requests to the serving loop, both schemes
        {"name": "serve_96", "path": "serve", "requests": 96, "most": 4096},
        # batch verification where nearly every batch is all valid (transactions already relayed)
        {"name": "rlc_valid_4096", "path": "rlc", "n": 262144, "batch": 4096, "bad_batches": 3},
        # the same with one invalid signature in every batch, which has to be found
        {"name": "rlc_one_bad_16384", "path": "rlc", "n": 524288, "batch": 16384, "bad_batches": 32},
        # a chain segment re-verified from host memory
        {"name": "ecdsa_host_1000003", "path": "host", "scheme": "ecdsa", "n": 1000003, "calls": 1},
        # the benchmark's headline batch
        {"name": "bip340_device_1048576", "path": "device", "scheme": "bip340", "n": _MAX_ITEMS},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["host", "host", "device", "device", "rows", "jobs", "serve", "rlc", "rlc"])
    if path == "host":
        n = _log_int(rng, 1, 1000003)
        return {"path": path, "scheme": rng.choice(["ecdsa", "bip340"]), "n": n, "calls": 16 if n < 64 else 1}
    if path == "device":
        return {"path": path, "scheme": rng.choice(["ecdsa", "bip340"]), "n": _log_int(rng, 100, 1000003)}
    if path == "rows":
        return {"path": path, "scheme": "ecdsa", "n": _log_int(rng, 50, 200000)}
    if path == "jobs":
        return {"path": path, "jobs": _log_int(rng, 20, 600), "most": _log_int(rng, 256, 8192)}
    if path == "serve":
        return {"path": path, "requests": _log_int(rng, 16, 128), "most": _log_int(rng, 256, 4096)}
    n, batch = _log_int(rng, 8192, 400000), _log_int(rng, 64, 16384)
    every = -(-n // min(n, batch))
    return {"path": path, "n": n, "batch": batch, "bad_batches": rng.choice([min(every, 3), every])}


@functools.lru_cache(None)
def _ctx():
    """The one context that a program keeps per GPU."""
    return uf.GpuContext(0)


@functools.lru_cache(None)
def _server():
    return uf.Server(_ctx())


def _keys(rng, n):
    # a leading byte below 0xFF keeps every key under the group order
    k = rng.integers(0, 256, (n, 32), dtype=np.uint8)
    k[:, 0] = rng.integers(1, 255, n, dtype=np.uint8)
    return k


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _signed(scheme, rng, sks):
    """Messages, public keys and signatures of `sks`, one row each, signed on the GPU (host arrays)."""
    ctx, n = _ctx(), len(sks)
    kind, pub = (0, 33) if scheme == "ecdsa" else (1, 32)
    msgs = rng.integers(0, 256, (n, 32), dtype=np.uint8)
    d_m, d_k, d_a = _dev(msgs), _dev(sks), _dev(rng.integers(0, 256, (n, 32), dtype=np.uint8))
    d_p = torch.empty(n * pub, dtype=torch.uint8, device="cuda")
    d_s = torch.empty(n * 64, dtype=torch.uint8, device="cuda")
    d_ok = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.sign_device(kind, d_m.data_ptr(), d_k.data_ptr(), d_a.data_ptr(), n, d_p.data_ptr(), d_s.data_ptr(),
                    d_ok.data_ptr())
    torch.cuda.synchronize()
    return msgs, d_p.cpu().numpy().reshape(n, pub), d_s.cpu().numpy().reshape(n, 64)


def _flip(rng, sigs, rows, lo=0):
    """One flipped bit in bytes lo..63 of each of `rows`."""
    bit = rng.integers(8 * lo, 512, len(rows))
    sigs[rows, bit >> 3] ^= (1 << (bit & 7)).astype(np.uint8)


def _few(rng, n):
    """The rows to spoil where a few signatures of a batch are bad: about 1 %, at least three."""
    return rng.choice(n, size=max(3, n // 100), replace=False)


def _mixed(rng, parts, most):
    """`parts` batches of log-uniform sizes 1..most, 70 % BIP-340 items, over a pool of keys, 0.5 % spoilt:
    (corpora by kind, kinds, starts, counts) as index ranges.  The sizes belong to the case, not to the seed."""
    of_case = np.random.default_rng([parts, most])
    sizes = np.exp(of_case.uniform(0, math.log(most), parts)).astype(np.int64).clip(1, most)
    n_e = of_case.binomial(sizes, 0.3)
    pool = _keys(rng, _KEY_POOL)
    weight = 1.0 / np.arange(1, _KEY_POOL + 1) ** 1.1
    corpora, kinds, starts, counts = {}, [], [], []
    for kind, per in ((0, n_e), (1, sizes - n_e)):
        n = max(1, int(per.sum()))
        m, p, s = _signed("bip340" if kind else "ecdsa", rng, pool[rng.choice(_KEY_POOL, n, p=weight / weight.sum())])
        _flip(rng, s, rng.choice(n, size=min(n, max(3, n // 200)), replace=False))
        corpora[kind] = (m, p, s)
        kinds.append(np.full(parts, kind))
        starts.append(np.concatenate([[0], np.cumsum(per)[:-1]]))
        counts.append(per)
    # each caller's ECDSA batch, then its BIP-340 batch
    return (corpora,) + tuple(np.stack(v, 1).reshape(-1) for v in (kinds, starts, counts))


def prepare(case, seed):
    rng = np.random.default_rng([seed, 256])
    path = case["path"]
    if path in ("jobs", "serve"):
        corpora, kinds, starts, counts = _mixed(rng, case["jobs" if path == "jobs" else "requests"], case["most"])
        if path == "jobs":
            _ctx()
            return {"path": path, "corpora": corpora, "ranges": (kinds, starts, counts)}
        _server()
        reqs = []
        for i in range(0, len(kinds), 2):
            reqs.append([(int(kinds[j]),) + tuple(a[starts[j]:starts[j] + counts[j]] for a in corpora[int(kinds[j])])
                         for j in (i, i + 1) if counts[j]])
        return {"path": path, "requests": reqs}
    n, calls = case["n"], case.get("calls", 1)
    m, p, s = _signed("bip340" if path == "rlc" else case["scheme"], rng, _keys(rng, n * calls))
    if path == "rlc":
        batch = case["batch"]
        first = np.arange(0, n, batch)
        first = rng.choice(first, size=case["bad_batches"], replace=False)
        _flip(rng, s, first + rng.integers(0, np.minimum(batch, n - first)), lo=32)
        return {"path": path, "n": n, "batch": batch, "seed32": rng.bytes(32), "d": [_dev(a) for a in (m, p, s)],
                "out": torch.zeros(n, dtype=torch.uint8, device="cuda")}
    _flip(rng, s, _few(rng, n * calls))
    if path == "rows":
        # libsecp's in-memory signature: r and s little-endian
        rows = np.concatenate([m, p, s[:, 31::-1], s[:, :31:-1]], axis=1)
        return {"path": path, "n": n, "rows": np.ascontiguousarray(rows), "fn": _rows_fn()}
    state = {"path": path, "scheme": case["scheme"], "n": n}
    if path == "host":
        return {**state, "h": [tuple(a[i:i + n] for a in (m, p, s)) for i in range(0, n * calls, n)]}
    return {**state, "d": [_dev(a) for a in (m, p, s)], "out": torch.zeros(n, dtype=torch.uint8, device="cuda")}


@functools.lru_cache(None)
def _rows_fn():
    fn = uf.load_library().ufsecp_gpu_ecdsa_verify_opaque_rows
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_void_p]
    return fn


def run(state):
    ctx, path = _ctx(), state["path"]
    if path == "host":
        call = ctx.ecdsa_verify_batch if state["scheme"] == "ecdsa" else ctx.schnorr_verify_batch
        return [call(*h) for h in state["h"]]
    if path == "device":
        call = ctx.ecdsa_verify_device if state["scheme"] == "ecdsa" else ctx.schnorr_verify_device
        m, p, s = state["d"]
        call(m.data_ptr(), p.data_ptr(), s.data_ptr(), state["n"], state["out"].data_ptr())
        return state["out"]
    if path == "rows":
        rows, out = state["rows"], np.zeros(state["n"], np.uint8)
        rc = state["fn"](ctx.handle, rows.ctypes.data, rows.shape[1], state["n"], out.ctypes.data)
        if rc != uf.UFSECP_OK:
            raise uf.UfsecpError(rc, "ufsecp_gpu_ecdsa_verify_opaque_rows")
        return out
    if path == "jobs":
        return ctx.verify_job_ranges(state["corpora"], *state["ranges"])
    if path == "serve":
        server = _server()
        ids = [server.submit(jobs) for jobs in state["requests"]]
        return np.concatenate([v for i in ids for v in server.wait(i)])
    m, p, s = state["d"]
    flags = ctx.schnorr_verify_rlc_device(m.data_ptr(), p.data_ptr(), s.data_ptr(), state["n"],
                                          state["out"].data_ptr(), batch_size=state["batch"], seed32=state["seed32"])
    return {"verdicts": state["out"], "batches": flags}


def _items(case):
    """Signatures of one pass and how many of them are ECDSA (on average for the drawn sizes of jobs and requests)."""
    if case["path"] in ("jobs", "serve"):
        n = case["jobs" if case["path"] == "jobs" else "requests"] * (case["most"] - 1) / math.log(case["most"])
        return n, 0.3 * n
    n = case["n"] * case.get("calls", 1)
    return n, n if case.get("scheme") == "ecdsa" else 0


def work(case):
    n, ecdsa = _items(case)
    macs = _RLC_MACS if case["path"] == "rlc" else _VERIFY_MACS
    return {"bytes": 129.0 * n + ecdsa, "flops": 2.0 * macs * n}
