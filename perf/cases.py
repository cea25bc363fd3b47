"""The work that programs built on this framework have it do, as timed cases.

Every case goes through a public entry point: proofs of single files, the
continuous-batching engine, verification, commitments of given witnesses, batched
ring products and the allocation-free file id.  Results are exact integers (proof
bytes, field elements, digests, verdicts).

Files are uniformly random bytes, as encrypted or compressed files are; ring
elements and witnesses are uniform in Z_q.  Like a long-running program, the
module keeps one context (and one engine or verifier service) per configuration.
"""
from __future__ import annotations

import ctypes
import functools
import math
import random

import numpy as np
import torch

import damascus000_gb300 as D

SYSTEM_SEED = D.DEFAULT_GENERATOR_SEED
EPOCH = D.DEFAULT_EPOCH_SEED
KIB, MIB = 1 << 10, 1 << 20


def listed():
    return [
        # the smallest whole proof (64 x 64 witness): stage latency and launches
        {"name": "prove_52k", "kind": "prove", "bytes": 53_248, "host": False},
        # an ordinary file handed over as host bytes
        {"name": "prove_1m_host", "kind": "prove", "bytes": MIB, "host": True},
        # a large file that is already in HBM (2048 x 2048 witness)
        {"name": "prove_16m", "kind": "prove", "bytes": 16 * MIB, "host": False},
        # a burst of files of all sizes at a prover service, each with its own generator seed
        {"name": "serve_files", "kind": "serve", "requests": 24, "lo": 50_000, "hi": 16 * MIB, "system_seed": False},
        # a deployment with one system seed: generator cache on, files in pinned host memory
        {"name": "serve_system_seed", "kind": "serve", "requests": 32, "lo": 50_000, "hi": 4 * MIB,
         "system_seed": True},
        # an auditor that checks proofs as they come, under per-file seeds
        {"name": "verify_each", "kind": "verify", "proofs": 12, "lo": 50_000, "hi": MIB, "service": False},
        # the streaming verifier over proofs of one system seed
        {"name": "verify_stream", "kind": "verify", "proofs": 24, "lo": 50_000, "hi": 16 * MIB, "service": True},
        # ring arithmetic as a building block: a handful of small products, the
        # usual batch, and large rings with an odd count
        {"name": "ring_5x64", "kind": "ring", "count": 5, "n": 64},
        {"name": "ring_4096x512", "kind": "ring", "count": 4096, "n": 512},
        {"name": "ring_301x2048", "kind": "ring", "count": 301, "n": 2048},
        # a commitment to a witness in host memory, fewer columns than a power of two
        {"name": "commit_777x512", "kind": "commit", "columns": 777, "n": 512},
        # the file id of a resident file whose length ends within a chunk
        {"name": "file_id_16m", "kind": "file_id", "bytes": 16 * MIB + 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prove", "prove", "serve", "verify", "ring", "ring", "commit", "file_id"])
    if kind == "prove":
        return {"kind": kind, "bytes": _log(rng, 1_000, 16 * MIB), "host": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(5, 24), "lo": 50_000, "hi": _log(rng, 100_000, 16 * MIB),
                "system_seed": rng.random() < 0.5}
    if kind == "verify":
        return {"kind": kind, "proofs": rng.randint(12, 24), "lo": 50_000, "hi": _log(rng, 100_000, MIB),
                "service": rng.random() < 0.5}
    if kind == "ring":
        n = 1 << rng.randint(3, 12)
        return {"kind": kind, "count": _log(rng, 1, (4096 * 512) // n), "n": n}
    if kind == "commit":
        n = 1 << rng.randint(4, 11)
        return {"kind": kind, "columns": _log(rng, 1, min(1024, (1024 * 512) // n)), "n": n}
    return {"kind": kind, "bytes": _log(rng, 1_000, 32 * MIB)}


# ------------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=None)
def _context(generator_cache: bool = False) -> D.Context:
    ctx = D.Context(0)
    if generator_cache:
        ctx.set_generator_cache(16 << 30)
    return ctx


@functools.lru_cache(maxsize=None)
def _engine(generator_cache: bool) -> D.Engine:
    return D.Engine(_context(generator_cache))


@functools.lru_cache(maxsize=None)
def _service() -> D.VerifyService:
    return D.VerifyService(_context())


# ------------------------------------------------------------------ inputs
def _random_bytes(gen, n):
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=gen)


def _random_elements(gen, *shape):
    """Uniform below 2^112 (above q = 2^112 - 75 with probability 2^-105): 16-byte words."""
    words = torch.randint(-(1 << 31), 1 << 31, (*shape, 4), dtype=torch.int32, device="cuda", generator=gen)
    words[..., 3] &= 0xFFFF
    return words


def _host(t) -> bytes:
    return t.cpu().numpy().tobytes()


def _sizes(count, lo, hi):
    """`count` file sizes spread evenly over the logarithm of [lo, hi]."""
    return [int(round(lo * (hi / lo) ** ((i + 0.5) / count))) for i in range(count)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "prove":
        s["ctx"] = _context()
        file = _random_bytes(gen, case["bytes"])
        s["file"] = _host(file) if case["host"] else file
        s["seed"] = _host(_random_bytes(gen, 32))
    elif kind == "serve":
        s["engine"] = _engine(case["system_seed"])
        sizes = _sizes(case["requests"], case["lo"], case["hi"])
        order = random.Random(len(sizes)).sample(range(len(sizes)), len(sizes))  # sizes arrive mixed
        s["pinned"] = case["system_seed"]
        s["requests"] = []
        for i in order:
            file = _random_bytes(gen, sizes[i])
            if case["system_seed"]:
                s["requests"].append((file.cpu().pin_memory(), SYSTEM_SEED))
            else:
                s["requests"].append((file, _host(_random_bytes(gen, 32))))
    elif kind == "verify":
        ctx = _context()
        s["ctx"], s["service"] = ctx, _service() if case["service"] else None
        s["proofs"] = []
        wrong = (_random_bytes(gen, case["proofs"]).cpu() < 85).tolist()  # a third open to another value
        for i, size in enumerate(_sizes(case["proofs"], case["lo"], case["hi"])):
            file = _random_bytes(gen, size)
            torch.cuda.synchronize()
            proof = ctx.prove_device(file.data_ptr(), size,
                                     SYSTEM_SEED if case["service"] else _host(_random_bytes(gen, 32)), EPOCH)
            s["proofs"].append(proof[:-16] + bytes([proof[-16] ^ 1]) + proof[-15:] if wrong[i] else proof)
    elif kind == "ring":
        s["ctx"] = _context()
        s["n"], s["count"] = case["n"], case["count"]
        s["a"] = _random_elements(gen, case["count"], case["n"])
        s["b"] = _random_elements(gen, case["count"], case["n"])
        s["out"] = torch.empty_like(s["a"])
    elif kind == "commit":
        s["ctx"] = _context()
        s["columns"], s["n"] = case["columns"], case["n"]
        s["witness"] = _host(_random_elements(gen, case["columns"], case["n"]))
        s["seed"] = _host(_random_bytes(gen, 32))
    else:
        s["lib"] = D.load()
        s["file"] = _random_bytes(gen, case["bytes"])
        s["out"] = torch.empty(32, dtype=torch.uint8, device="cuda")
    return s


# ------------------------------------------------------------------ one pass
def _array(b: bytes):
    return np.frombuffer(b, dtype=np.uint8)


def run(s):
    kind = s["kind"]
    if kind == "prove":
        f = s["file"]
        if isinstance(f, bytes):
            return _array(s["ctx"].prove(f, s["seed"], EPOCH))
        return _array(s["ctx"].prove_device(f.data_ptr(), f.numel(), s["seed"], EPOCH))
    if kind == "serve":
        eng = s["engine"]
        submit = eng.submit_borrowed if s["pinned"] else eng.submit_device
        tickets = [submit(f.data_ptr(), f.numel(), seed, EPOCH) for f, seed in s["requests"]]
        done = {t: proof for t, proof, _ in eng.as_completed(tickets)}
        return [_array(done[t]) for t in tickets]
    if kind == "verify":
        if s["service"] is not None:
            return s["service"].verify_batch(s["proofs"], EPOCH)
        return [s["ctx"].verify(p, EPOCH) for p in s["proofs"]]
    if kind == "ring":
        s["ctx"].ring_mul_batch_device(s["a"].data_ptr(), s["b"].data_ptr(), s["out"].data_ptr(), s["n"], s["count"])
        return s["out"]
    if kind == "commit":
        return _array(s["ctx"].commit_witness(s["witness"], s["columns"], s["n"], s["seed"]))
    rc = s["lib"].damascus_file_id_noalloc(ctypes.c_void_p(s["file"].data_ptr()), s["file"].numel(),
                                           ctypes.c_void_p(s["out"].data_ptr()),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise D.DamascusError(rc, "file_id_noalloc")
    return s["out"]


def exact(case, seed):
    """No floating-point output anywhere: every result is bytes or whole numbers."""
    return None


# ------------------------------------------------------------------ the work of one pass
HASH_OPS = 7 * 8 * 14  # 32-bit operations of one BLAKE3 compression
MUL_OPS = 2 * 16       # 32-bit multiply-adds of one 112 x 112-bit product


def _proof_work(n_bytes, proving):
    """(bytes, operations) of one proof: the file or the proof in, the proof out, one
    compression per generator coefficient, and per coefficient of the (halving)
    family the products of the folds and, for the prover, of the three sums."""
    d, dim = D.layout_for_byte_len(n_bytes)
    proof = D.proof_size(n_bytes)
    family = 8 * dim * dim
    products = family * (4 if proving else 1)
    ops = family * HASH_OPS + products * MUL_OPS + (proof + (n_bytes if proving else 0)) / 64 * HASH_OPS
    return (n_bytes if proving else 0) + proof, ops


def work(case):
    kind = case["kind"]
    if kind == "prove":
        b, f = _proof_work(case["bytes"], True)
    elif kind in ("serve", "verify"):
        each = [_proof_work(n, kind == "serve")
                for n in _sizes(case["requests" if kind == "serve" else "proofs"], case["lo"], case["hi"])]
        b, f = sum(x for x, _ in each), sum(y for _, y in each)
    elif kind == "ring":
        n, count = case["n"], case["count"]
        b, f = 3 * 16 * n * count, count * n * (1 + math.log2(n)) * MUL_OPS
    elif kind == "commit":
        n, cols = case["n"], case["columns"]
        b = 16 * n * (cols + 8)
        f = 8 * n * cols * (HASH_OPS + MUL_OPS * (1 + math.log2(n)))
    else:
        b, f = case["bytes"] + 32, case["bytes"] / 64 * HASH_OPS
    return {"bytes": float(b), "flops": float(f)}
