"""The measured work of the prover: what its users call, over the sizes they call it at.

Every pass goes through the Python binding of the C ABI
(flock-challenge-multi_b200/flockgpu.py) with host inputs, as the reference's
callers hand them over, and returns the whole result (the proof bundle's
bytes, the verifier's verdict).

A user's program keeps a context per device and a setup per statement size,
so `prepare` builds those with the inputs, and `run` is one call.  All outputs
are bytes, so they have to be equal, not close; there is nothing to evaluate
in 64 bits and this file has no `exact`.

Sizes are the repository's own: 2^10 and 2^18 compressions are the plain
proofs of its benchmark, 2^12..2^18 its batched jobs, the SHA-256 and Keccak
counts lie among those of the reference's benches, and counts that are no
power of two exercise the padding slots.
"""
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "flock-challenge-multi_b200"))
import flockgpu  # noqa: E402

_context = []


def _ctx():
    """The process's one context (a program keeps one per device)."""
    if not _context:
        _context.append(flockgpu.Context(0))
    return _context[0]


def listed():
    return [
        # the smallest plain proof of the benchmark: latency, launches and host round trips
        {"name": "blake3_1k", "kind": "blake3", "n": 1 << 10, "hashes": "blake3"},
        # a caller's own list of compressions, no power of two, with the reference's default
        # hash (SHA-256) behind the Merkle trees and the transcript
        {"name": "blake3_3001_sha256_hashes", "kind": "blake3", "n": 3001, "hashes": "sha256"},
        # an ordinary proof
        {"name": "blake3_16k", "kind": "blake3", "n": 1 << 14, "hashes": "blake3"},
        # a large ragged proof: 31,071 of its 131,072 slots are padding
        {"name": "blake3_100001", "kind": "blake3", "n": 100001, "hashes": "blake3"},
        # the headline: one proof of 2^18 compressions
        {"name": "blake3_256k", "kind": "blake3", "n": 1 << 18, "hashes": "blake3"},
        # a hash chain of the command-line tool
        {"name": "blake3_chain_8k", "kind": "chain", "n": 1 << 13},
        # SHA-256 compressions, a ragged count
        {"name": "sha256_5000", "kind": "sha256", "n": 5000, "hashes": "blake3"},
        # SHA-256 Merkle paths: 16 paths of 256 hashes
        {"name": "sha256_paths_4k", "kind": "merkle", "n": 1 << 12, "path_log": 4},
        # Keccak permutations, the single and the 3-wide encoder
        {"name": "keccak_3000", "kind": "keccak", "n": 3000, "width": 1},
        {"name": "keccak3_24k", "kind": "keccak", "n": 24576, "width": 3},
        # a server's batch: uneven jobs drawn log-uniform, proved together
        {"name": "batch_24_jobs", "kind": "batch", "jobs": 24, "lo": 10, "hi": 16},
        # a server that checks each proof before it hands it out
        {"name": "checked_2k", "kind": "checked", "n": 1 << 11},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["blake3", "blake3", "blake3", "chain", "sha256", "merkle", "keccak", "batch", "checked"])
    if kind == "blake3":
        return {"kind": kind, "n": _log_int(rng, 600, 1 << 18), "hashes": rng.choice(["blake3", "blake3", "sha256"])}
    if kind == "chain":
        return {"kind": kind, "n": 1 << rng.randint(9, 17)}
    if kind == "sha256":
        return {"kind": kind, "n": _log_int(rng, 300, 100000), "hashes": rng.choice(["blake3", "sha256"])}
    if kind == "merkle":
        n_log = rng.randint(8, 15)
        return {"kind": kind, "n": 1 << n_log, "path_log": rng.randint(0, n_log)}
    if kind == "keccak":
        return {"kind": kind, "n": _log_int(rng, 150, 50000), "width": rng.choice([1, 3])}
    if kind == "batch":
        lo = rng.randint(9, 11)
        return {"kind": kind, "jobs": rng.randint(5, 24), "lo": lo, "hi": lo + rng.randint(1, 4)}
    return {"kind": kind, "n": 1 << rng.randint(9, 16)}


def _blake3_blocks(rng, n):
    """(n, 25) u32: cv, message and counter, all uniform."""
    return rng.integers(0, 1 << 32, size=(n, 25), dtype=np.uint32)


def _pinned(a):
    p = flockgpu.PinnedArray(a.shape, a.dtype)
    p.array[...] = a
    return p


def _job_logs(case):
    """Job sizes spread evenly over the logarithm of the range, in a fixed shuffled order."""
    k = case["jobs"]
    logs = [case["lo"] + round((case["hi"] - case["lo"]) * i / max(k - 1, 1)) for i in range(k)]
    order = np.random.default_rng(7).permutation(k)
    return [logs[i] for i in order]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    ctx, kind = _ctx(), case["kind"]
    st = {"kind": kind, "ctx": ctx}
    if kind == "blake3":
        n, h = case["n"], case["hashes"]
        st["pow2"] = n & (n - 1) == 0
        if st["pow2"]:
            st["prover"] = flockgpu.Prover(ctx, n.bit_length() - 1, merkle_hash=h, transcript=h)
            st["in"] = _pinned(_blake3_blocks(rng, n))
        else:
            st["prover"] = flockgpu.Prover(ctx, n_blocks=n, merkle_hash=h, transcript=h)
            st["in"] = _pinned(flockgpu.to_records(_blake3_blocks(rng, n)))
    elif kind == "chain":
        st["prover"] = flockgpu.Prover(ctx, case["n"].bit_length() - 1)
        st["in"] = _pinned(flockgpu.chain_blocks(seed, case["n"]))
    elif kind == "sha256":
        st["prover"] = flockgpu.Sha256Prover(ctx, case["n"], merkle_hash=case["hashes"], transcript=case["hashes"])
        st["in"] = _pinned(flockgpu.sha256_bench_inputs(case["n"], seed))
    elif kind == "merkle":
        st["prover"] = flockgpu.Sha256Prover(ctx, case["n"])
        st["path_log"] = case["path_log"]
        st["in"], st["bits"], _, _ = flockgpu.sha256_merkle_inputs(case["n"].bit_length() - 1, case["path_log"], seed)
    elif kind == "keccak":
        st["prover"] = flockgpu.KeccakProver(ctx, case["n"], width=case["width"])
        st["in"] = _pinned(flockgpu.keccak_bench_inputs(case["n"], seed))
    elif kind == "batch":
        # half of the jobs bring their compressions, half a generator seed
        st["jobs"] = [(lg, _blake3_blocks(rng, 1 << lg) if i % 2 else int(rng.integers(1 << 62)))
                      for i, lg in enumerate(_job_logs(case))]
    else:
        st["prover"] = flockgpu.Prover(ctx, case["n"].bit_length() - 1)
        st["in"] = _pinned(_blake3_blocks(rng, case["n"]))
    st["out"] = [np.zeros(flockgpu.MAX_PROOF_BYTES, np.uint8) for _ in range(case.get("jobs", 1))]
    return st


def _keep(st, bundle, i=0):
    """A bundle's length depends on its openings, so it is returned as its
    length and its bytes in a buffer of the largest allowed size."""
    out = st["out"][i]
    out[: len(bundle)] = np.frombuffer(bundle, np.uint8)
    out[len(bundle):] = 0
    return [len(bundle), out]


def run(st):
    kind = st["kind"]
    if kind == "blake3":
        x = st["in"].array
        return _keep(st, st["prover"].prove_blocks(x) if st["pow2"] else st["prover"].prove_compressions(x))
    if kind == "chain":
        return _keep(st, st["prover"].prove_chain(st["in"].array))
    if kind in ("sha256", "keccak"):
        return _keep(st, st["prover"].prove(st["in"].array))
    if kind == "merkle":
        return _keep(st, st["prover"].prove_merkle(st["in"], st["bits"], st["path_log"]))
    if kind == "batch":
        return [_keep(st, r["bytes"], i) for i, r in enumerate(st["ctx"].prove_batch(st["jobs"]))]
    bundle = st["prover"].prove_blocks(st["in"].array)
    return _keep(st, bundle) + [int(st["prover"].verify(bundle) == "")]


# Block size (log2 of its bits) and input bytes per compression of each statement.
_SHAPE = {"blake3": (14, 100), "checked": (14, 100), "chain": (14, 112), "sha256": (15, 96), "merkle": (15, 97)}
# One field product as shift-and-XOR steps over four 32-bit words.
_PRODUCT = 512


def _proof_work(k_log, n_slots, in_bytes):
    """Bytes in and out of one proof, and the 32-bit operations of its three
    largest parts: the additive NTT of the commitment (2^(m-12) positions of
    64 values at rate 1/2), the 2^(m-6)-row zerocheck and the openings' folds
    (about ten products per 128-bit word of the witness), and the BLAKE3 tree
    over the codeword's 1 KiB leaves (16 + 1 compressions of 800 operations)."""
    m = k_log + max(3, (n_slots - 1).bit_length())
    words = 1 << (m - 7)
    ntt = (m - 13) * words
    proof = 270000 + 20000 * max(0, m - 24)
    return {"bytes": in_bytes + proof, "flops": (ntt + 10 * words) * _PRODUCT + (words // 32) * 17 * 800}


def work(case):
    kind = case["kind"]
    if kind in _SHAPE:
        k_log, b = _SHAPE[kind]
        return _proof_work(k_log, case["n"], b * case["n"])
    if kind == "keccak":
        blocks = -(-case["n"] // case["width"])
        return _proof_work(16 if case["width"] == 1 else 17, blocks, 200 * case["n"])
    if kind == "batch":
        ws = [_proof_work(14, 1 << lg, (100 << lg) if i % 2 else 8) for i, lg in enumerate(_job_logs(case))]
    return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
