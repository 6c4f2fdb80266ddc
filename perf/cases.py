"""Timing cases of the prover: what programs call it for, through the package's public entry points.

A case names an operation and its sizes. The provers and servers a program keeps
for its lifetime (their buffers grow to the largest size seen) are made once per
size and kept here too; a state holds one call's inputs.
"""
import functools

import numpy as np
import torch

import flock_challenge_gb300 as F

K_LOG = 14  # witness bits per compression (log2)


def listed():
    return [
        # One small request as a service meets it: 256 compressions is the
        # smallest batch the proof system's parameters cover. Latency only.
        {"name": "prove_256", "op": "prove", "n": 256},
        # A batch that is no power of two (the prover pads it to 2^13 slots).
        {"name": "prove_ragged_5000", "op": "prove", "n": 5000},
        # The reference worker's timed path (seed -> inputs -> proof) at its
        # small benchmark size.
        {"name": "prove_seed_2e14", "op": "prove_seed", "log2": 14},
        # The reference's headline benchmark: 2^18 compressions in host memory.
        {"name": "prove_2e18", "op": "prove", "n": 1 << 18},
        # The largest requests of the served mix, records already on the GPU.
        {"name": "prove_device_2e20", "op": "prove_device", "n": 1 << 20},
        # A hash chain of 2^12 links (flock_chain's relation).
        {"name": "prove_chain_2e12", "op": "prove_chain", "log2": 12},
        # What the receiver of a proof does, continuing its own transcript.
        {"name": "verify_2e16", "op": "verify", "log2": 16},
        # Mixed requests proven through the server's concurrent workers.
        {"name": "batch_12x_2e10_2e15", "op": "batch", "count": 12, "lo": 10, "hi": 15},
        # The commitment seam alone (witness in, codeword, tree and root out)
        # as the prover's first step calls it: 2^16 compressions, rate 1/2.
        {"name": "commit_64x2e18", "op": "commit", "m": 30, "rate": 1, "batch": 6},
        # The commitment microbenchmark's shape: 256 columns, rate 1/4, 4 KiB
        # leaves, at 2^15 rows.
        {"name": "commit_256x2e15", "op": "commit", "m": 30, "rate": 2, "batch": 8},
        # One transform of 8 lanes, the recursive levels' code shape.
        {"name": "ntt_8x2e16", "op": "ntt", "log_d": 16, "lanes": 3, "start": 2},
        # Witness generation alone, with the a, b planes and the byte stripe.
        {"name": "witness_100000", "op": "witness", "n": 100000},
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over its logarithm in [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["prove", "prove", "prove_seed", "prove_device", "prove_chain", "verify", "batch", "commit",
                     "commit", "ntt", "witness"])
    if op in ("prove", "prove_device"):
        return {"op": op, "n": _log(rng, 200, 1 << 19) | 1}
    if op == "prove_seed":
        return {"op": op, "log2": rng.randint(8, 18), "tag": rng.randrange(1 << 20)}
    if op in ("prove_chain", "verify"):
        return {"op": op, "log2": rng.randint(8, 16), "tag": rng.randrange(1 << 20)}
    if op == "batch":
        lo = rng.randint(8, 12)
        return {"op": op, "count": rng.randint(4, 16), "lo": lo, "hi": lo + rng.randint(0, 4)}
    if op == "commit":
        batch = rng.randint(4, 8)
        return {"op": op, "m": rng.randint(max(20, batch + 11), 31), "rate": rng.randint(1, 3), "batch": batch}
    if op == "ntt":
        lanes = rng.randint(3, 8)
        return {"op": op, "log_d": rng.randint(4, 24 - lanes), "lanes": lanes, "start": rng.randint(0, 3)}
    return {"op": op, "n": _log(rng, 8, 1 << 18) | 1}


def _records(n, seed):
    """n compressions of the benchmark's distribution: random 32-bit words, whole blocks, flags 11."""
    rng = np.random.default_rng(seed)
    words = rng.integers(0, 1 << 32, size=(n, 25), dtype=np.uint32)
    rec = np.zeros(n, F.COMPRESSION_DTYPE)
    rec["cv"] = words[:, :8]
    rec["m"] = words[:, 8:24]
    rec["counter"] = words[:, 24]
    rec["block_len"] = 64
    rec["flags"] = 11
    return rec


def _random_bytes(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-(1 << 63), (1 << 63) - 1, (n // 8,), dtype=torch.int64, device="cuda", generator=g).view(
        torch.uint8)


@functools.lru_cache(maxsize=None)
def _setup(n):
    return F.Blake3Setup(n)


@functools.lru_cache(maxsize=None)
def _server():
    return F.Server(workers=4)


@functools.lru_cache(maxsize=None)
def _context():
    return F.Context(0)


def prepare(case, seed):
    op, s = case["op"], dict(case)
    seed += case.get("tag", 0)  # drawn cases of one size: other inputs
    if op == "prove":
        s["setup"], s["blocks"] = _setup(case["n"]), _records(case["n"], seed)
    elif op == "prove_device":
        s["setup"] = _setup(case["n"])
        s["blocks"] = torch.from_numpy(_records(case["n"], seed).view(np.uint8)).cuda()
    elif op == "prove_seed":
        s["setup"], s["seed"] = _setup(1 << case["log2"]), seed
    elif op == "prove_chain":
        s["setup"], s["blocks"] = _setup(1 << case["log2"]), F.chain_inputs(1 << case["log2"], seed)
    elif op == "verify":
        s["setup"] = _setup(1 << case["log2"])
        s["proof"] = s["setup"].prove_seed(seed)
    elif op == "batch":
        rng = np.random.default_rng(seed)
        s["server"] = _server()
        s["sizes"] = [case["lo"] + i % (case["hi"] - case["lo"] + 1) for i in range(case["count"])]
        s["seeds"] = [int(x) for x in rng.integers(0, 1 << 62, size=case["count"])]
    elif op == "commit":
        s["ctx"], s["z"] = _context(), _random_bytes((1 << case["m"]) // 8, seed)
    elif op == "ntt":
        s["ctx"], s["data"] = _context(), _random_bytes(16 << (case["log_d"] + case["lanes"]), seed)
    elif op == "witness":
        s["blocks"] = torch.from_numpy(_records(case["n"], seed).view(np.uint8)).cuda()
        s["n_log"] = max(3, (case["n"] - 1).bit_length())
    return s


def _array(b):
    return np.frombuffer(b, np.uint8)


PROOF_CAP = 1 << 19


def _keep(s, proofs):
    """The proofs in the caller's buffers (a proof's size depends on its openings), and their sizes."""
    bufs = s.get("out") or s.setdefault("out", [np.zeros(PROOF_CAP, np.uint8) for _ in proofs])
    for buf, p in zip(bufs, proofs):
        buf[:len(p)] = _array(p)
    return [*bufs, np.array([len(p) for p in proofs])]


def run(s):
    op = s["op"]
    if op == "prove":
        return _keep(s, [s["setup"].prove_fast(s["blocks"])])
    if op == "prove_device":
        return _keep(s, [s["setup"].prove_device(s["blocks"])])
    if op == "prove_seed":
        return _keep(s, [s["setup"].prove_seed(s["seed"])])
    if op == "prove_chain":
        return _keep(s, [s["setup"].prove_chain(s["blocks"])])
    if op == "verify":
        tr = F.FsChallenger()
        ok = F.verify(s["proof"], ctx=s["setup"].ctx, challenger=tr)
        # the transcript's next challenge: a function of the whole replay
        return [ok, np.array(tr.sample_f128(), np.uint64).view(np.uint8)]
    if op == "batch":
        return _keep(s, s["server"].prove_batch(s["sizes"], s["seeds"]))
    if op == "commit":
        root, cw, tree = F.commit(s["ctx"], s["z"], s["m"], s["rate"], s["batch"])
        return [_array(root), cw, tree]
    if op == "ntt":
        F.ntt(s["ctx"], s["data"], s["log_d"], s["lanes"], s["start"])
        return s["data"]
    z, a, b, stripe = F.generate_witness(s["blocks"], s["n"], s["n_log"])
    return [z, a, b, stripe]


def _proof_bytes(n):
    """About the size of a proof of n compressions (272 kB at 2^8, 437 kB at 2^18)."""
    return 272_000 + 16_500 * (max(8, (n - 1).bit_length()) - 8)


def work(case):
    """Bytes of the inputs and outputs. The arithmetic is GF(2^128) and 32-bit
    integer work: no floating-point operation is needed."""
    op = case["op"]
    if op in ("prove", "prove_device"):
        return {"bytes": 112 * case["n"] + _proof_bytes(case["n"]), "flops": 0}
    if op == "prove_seed":
        return {"bytes": _proof_bytes(1 << case["log2"]), "flops": 0}
    if op == "prove_chain":
        return {"bytes": (112 << case["log2"]) + _proof_bytes(1 << case["log2"]), "flops": 0}
    if op == "verify":
        return {"bytes": _proof_bytes(1 << case["log2"]), "flops": 0}
    if op == "batch":
        sizes = [case["lo"] + i % (case["hi"] - case["lo"] + 1) for i in range(case["count"])]
        return {"bytes": sum(_proof_bytes(1 << k) for k in sizes), "flops": 0}
    if op == "commit":
        message = (1 << case["m"]) // 8
        positions = 1 << (case["m"] - 7 - case["batch"] + case["rate"])
        return {"bytes": message + (message << case["rate"]) + 32 * (2 * positions - 1), "flops": 0}
    if op == "ntt":
        return {"bytes": 2 * (16 << (case["log_d"] + case["lanes"])), "flops": 0}
    slots = 1 << max(3, (case["n"] - 1).bit_length())
    return {"bytes": 112 * case["n"] + 4 * (slots << K_LOG) // 8, "flops": 0}


def exact(case, seed):
    """Every output is bytes, which are compared as they are."""
    return None
