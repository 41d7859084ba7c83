"""The work this framework is measured by, through its public entry points.

A case is one call (or one staged group of calls) a user's program makes: a proof of a SHA-256
statement, its verification, a batch of proofs, or one of the reductions that the library also
exports by itself (the grand-product GKR and the post-GKR sumcheck). Outputs are proof bytes,
transcript bytes and field elements held as whole numbers: all exact, so there is nothing to
compare with in floating point.
"""
import ctypes
import os
import random

import numpy as np
import torch

# A program that initialises CUDA before it loads the library asks for the hardware queues that
# the library would ask for otherwise ("Batch and serving").
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import bitz_b200 as bz  # noqa: E402
from bitz_b200 import _lib, statements  # noqa: E402

_U64P = ctypes.POINTER(ctypes.c_uint64)


def listed():
    return [
        # one 64-byte block with its chaining value: the smallest statement, launches and rounds only
        {"name": "prove-compression", "op": "prove", "kind": "sha256-compression", "blocks": 1, "security": 100},
        # the headline workload: a chain of 64 blocks
        {"name": "prove-chain-64", "op": "prove", "kind": "sha256-chain", "blocks": 64, "security": 100},
        # a 2 KiB message through the reference's three calls (witness, commit, prove), 128 bits
        {"name": "staged-2kb-128", "op": "staged", "kind": "sha256-2kb", "blocks": 32, "security": 128},
        # the large configuration: a chain of 1024 blocks at 128 bits
        {"name": "prove-chain-1024-128", "op": "prove", "kind": "sha256-chain", "blocks": 1024, "security": 128},
        # a padded message of an odd length, the serving mix's larger half
        {"name": "prove-aligned-201", "op": "prove", "kind": "sha256-block-aligned", "blocks": 201, "security": 100},
        # the receiving side of the headline workload
        {"name": "verify-chain-64", "op": "verify", "kind": "sha256-chain", "blocks": 64, "security": 100},
        # many independent messages of 0 to 32 blocks at once, as the batched workload has them
        {"name": "batch-48", "op": "batch", "count": 48, "max_blocks": 32, "mix": 3, "security": 100},
        # the grand-product GKR by itself on device tables: a small claim and the largest statement's
        {"name": "gkr-10", "op": "gkr", "log_cols": 10, "security": 100},
        {"name": "gkr-18-128", "op": "gkr", "log_cols": 18, "security": 128},
        # the product tree's output layer from host arrays
        {"name": "gkr-outputs-15", "op": "gkr_outputs", "log_cols": 15},
        # the post-GKR sumcheck on a product claim (128 row weights by 2^18 column weights)
        {"name": "post-gkr-7x18", "op": "post_gkr", "log_rows": 7, "log_cols": 18, "security": 100},
        # the same sumcheck without allocation, on the caller's stream
        {"name": "post-gkr-noalloc-17", "op": "post_gkr_noalloc", "log_rows": 17, "log_cols": 0, "security": 100},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(lo * (hi / lo) ** rng.random() * rng.uniform(1.0, 1.02))))


def draw(rng):
    op = rng.choice(["prove", "prove", "staged", "verify", "batch", "gkr", "gkr", "gkr_outputs", "post_gkr", "post_gkr", "post_gkr_noalloc"])
    security = rng.choice([100, 128])
    if op in ("prove", "staged", "verify"):
        kind = rng.choice(["sha256-chain", "sha256-block-aligned"] + (["sha256-compression"] if op == "staged" else []))
        blocks = 1 if kind == "sha256-compression" else _log_uniform(rng, 1, 512 if op == "prove" else 128)
        return {"op": op, "kind": kind, "blocks": blocks, "security": security}
    if op == "batch":
        return {"op": op, "count": _log_uniform(rng, 4, 48), "max_blocks": rng.randint(2, 32), "mix": rng.randrange(1 << 20), "security": security}
    if op == "gkr":
        return {"op": op, "log_cols": rng.randint(4, 18), "security": security}
    if op == "gkr_outputs":
        return {"op": op, "log_cols": rng.randint(4, 16)}
    if op == "post_gkr_noalloc":
        m = rng.randint(9, 20)
    else:
        m = rng.randint(9, 25)
    log_rows = rng.randint(7, m)
    return {"op": op, "log_rows": log_rows, "log_cols": m - log_rows, "security": security}


# ------------------------------------------------------------------- inputs


def _statement(kind, blocks, seed):
    state = statements.random_state(seed) if kind == "sha256-compression" else None
    inputs, outputs, _ = statements.instance(kind, blocks, seed, state)
    return inputs, outputs


def _elements(gen, *shape):
    """Uniform GF(2^128) elements on the device: int64 (..., 2) holding (lo, hi)."""
    return torch.randint(-2**63, 2**63 - 1, (*shape, 2), dtype=torch.int64, device="cuda", generator=gen)


def _xor_over(x):
    """XOR of x over its first dimension (a power of two long)."""
    while x.shape[0] > 1:
        h = x.shape[0] // 2
        x = x[:h] ^ x[h:]
    return x[0]


def _gf_mul(a, b):
    """Products in GF(2^128) = F_2[X]/(X^128 + X^7 + X^2 + X + 1), element by element."""
    lo, hi = torch.zeros_like(a[..., 0]), torch.zeros_like(a[..., 0])
    for i in range(127, -1, -1):
        top = -((hi >> 63) & 1)
        hi = (hi << 1) | ((lo >> 63) & 1)
        lo = (lo << 1) ^ (top & 0x87)
        bit = -((b[..., i >> 6] >> (i & 63)) & 1)
        lo = lo ^ (bit & a[..., 0])
        hi = hi ^ (bit & a[..., 1])
    return torch.stack((lo, hi), dim=-1)


def _weighted_sum(rows, cols, packed):
    """<rows (x) cols, f> over the bits f of the packed words."""
    shift = torch.arange(64, device="cuda")
    bits = ((packed.unsqueeze(-1) >> shift) & 1).reshape(cols.shape[0], rows.shape[0])
    per_col = _xor_over((-bits.t()).unsqueeze(-1) & rows.unsqueeze(1))
    return _xor_over(_gf_mul(per_col, cols))


def _words(t):
    """A device tensor's 64-bit words as a ctypes array."""
    v = [int(x) & (2**64 - 1) for x in t.reshape(-1).tolist()]
    return (ctypes.c_uint64 * len(v))(*v)


def prepare(case, seed):
    op = case["op"]
    if op in ("prove", "staged", "verify"):
        inputs, outputs = _statement(case["kind"], case["blocks"], seed)
        ps = bz.CircuitProofSystem(case["kind"], inputs, outputs, case["security"])
        state = {"op": op, "ps": ps, "inputs": inputs}
        if op == "verify":
            state["proof"] = ps.prove()[0]
        return state
    if op == "batch":
        # lengths are the case's (uniform over 0..max_blocks), the messages the seed's
        lengths = random.Random(case["mix"])
        blocks = [lengths.randint(0, case["max_blocks"]) for _ in range(case["count"])]
        kind = "sha256-block-aligned"
        return {"op": op, "systems": [bz.CircuitProofSystem(kind, *_statement(kind, k, seed + 1000003 * i), case["security"])
                                      for i, k in enumerate(blocks)]}
    if op == "gkr_outputs":
        rng = np.random.default_rng(seed)
        draw64 = lambda n: rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64)  # noqa: E731
        return {"op": op, "images": draw64(128), "columns": draw64(1 << case["log_cols"])}
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if op == "gkr":
        s = case["log_cols"]
        state = {"op": op, "log_cols": s, "security": case["security"], "images": _elements(gen, 128),
                 "columns": _elements(gen, 1 << s), "zeta": _words(_elements(gen, s))}
    else:
        t, s = case["log_rows"], case["log_cols"]
        rows, cols = _elements(gen, 1 << t), _elements(gen, 1 << s)
        packed = _elements(gen, 1 << (t + s - 7))
        state = {"op": op, "log_rows": t, "log_cols": s, "security": case["security"], "rows": rows, "cols": cols,
                 "packed": packed, "target": _words(_weighted_sum(rows, cols, packed))}
    torch.cuda.synchronize()  # the library proves on streams of its own
    return state


# --------------------------------------------------------------------- work


def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def _ok(status):
    if status != 0:
        raise RuntimeError("status %d: %r" % (status, _lib.load().bitz_last_error()))


def _run_gkr(state):
    s = state["log_cols"]
    transcript = bz.build_prover(b"bitz/perf", b"gkr")
    point, claim = np.zeros((s + 7, 2), dtype=np.uint64), np.zeros(2, dtype=np.uint64)
    _ok(_lib.load().bitz_gkr_prove_dev(
        state["images"].data_ptr(), state["columns"].data_ptr(), s, state["zeta"], state["security"], transcript.handle,
        point.ctypes.data_as(_U64P), claim.ctypes.data_as(_U64P)))
    return {"point": point, "claim": claim, "narg": _bytes(transcript.narg())}


def _run_post_gkr(state):
    t, s = state["log_rows"], state["log_cols"]
    transcript = bz.build_prover(b"bitz/perf", b"post-gkr")
    point, value = np.zeros((t + s, 2), dtype=np.uint64), np.zeros(2, dtype=np.uint64)
    args = [state["rows"].data_ptr(), t, state["cols"].data_ptr(), s, state["target"], state["packed"].data_ptr(),
            state["security"], transcript.handle]
    out = [point.ctypes.data_as(_U64P), value.ctypes.data_as(_U64P)]
    if state["op"] == "post_gkr_noalloc":
        _ok(_lib.load().bitz_post_gkr_prove_noalloc(*args, torch.cuda.current_stream().cuda_stream, *out))
    else:
        _ok(_lib.load().bitz_post_gkr_prove_dev(*args, *out))
    return {"point": point, "value": value, "narg": _bytes(transcript.narg())}


def run(state):
    op = state["op"]
    if op == "prove":
        return _bytes(state["ps"].prove()[0])
    if op == "staged":
        ps = state["ps"]
        witness = ps.witness(state["inputs"])
        return _bytes(ps.prove(witness, ps.commit(witness))[0])
    if op == "verify":
        state["ps"].verify(state["proof"])  # raises unless the proof is accepted
        return {"accepted": 1, "proof": _bytes(state["proof"])}
    if op == "batch":
        return [_bytes(p) for p in bz.batch_prove(state["systems"])[0]]
    if op == "gkr":
        return _run_gkr(state)
    if op == "gkr_outputs":
        return bz.gkr_outputs(state["images"], state["columns"])
    return _run_post_gkr(state)


# A compression allocates 20,456 bits of h and 6,376 of f; the statement's constraints and the
# proof are a few hundred kilobytes and 16 bytes per packed column.
_H_BITS, _F_BITS, _PROOF_BYTES = 20456, 6376, 330_000


def _proof_work(kind, blocks):
    if kind in ("sha256-block-aligned", "sha256-2kb"):
        blocks += 1
    cols = 128
    while cols * 128 < blocks * _H_BITS:
        cols *= 2
    # in: the statement's bits, one byte each; out: the proof. Field products: the product tree
    # (127 a column) and its seven sumchecks (about 8 per leaf), and the committed bits' sumcheck
    # (about 4 per bit)
    return {"bytes": 512 * blocks + 256 + _PROOF_BYTES + 16 * cols, "flops": 127 * cols + 8 * 128 * cols + 4 * _F_BITS * blocks}


def work(case):
    """Bytes: the inputs once and the outputs once. Operations: the field products that the
    reduction is made of, one each (they are exact integer work, not floating point)."""
    op = case["op"]
    if op in ("prove", "staged"):
        return _proof_work(case["kind"], case["blocks"])
    if op == "verify":
        w = _proof_work(case["kind"], case["blocks"])
        return {"bytes": w["bytes"], "flops": 4 * _F_BITS * case["blocks"]}
    if op == "batch":
        one = _proof_work("sha256-block-aligned", case["max_blocks"] // 2)
        return {k: case["count"] * v for k, v in one.items()}
    if op in ("gkr", "gkr_outputs"):
        n = 1 << case["log_cols"]
        if op == "gkr_outputs":
            return {"bytes": 128 * 16 + 16 * n + 16 * n, "flops": 127 * n}
        return {"bytes": 128 * 16 + 16 * n, "flops": 127 * n + 8 * 128 * n}
    m = case["log_rows"] + case["log_cols"]
    return {"bytes": (16 << case["log_rows"]) + (16 << case["log_cols"]) + (1 << m) // 8, "flops": 4 << m}
