"""The measured workloads of the prover: what a program that proves, verifies and serves with
this package has it do, each as one pass through the package's public entry points.

Sizes are powers of two of rows by the nature of the protocol; the ranges below run from the
smallest proofs, where launches, round trips and the transcript's latency count, to the plain
2^20-row proof and the 2^24-value sumcheck, and what is irregular in use varies with them: the
univariate skip, the code rate, the security level, the number and mix of proofs in a batch.

A case is a dict of plain values; "path" names the entry point:

  witness    AirTable.prove_witness: the witness is resident in device memory
  inputs     Witness.generate + AirTable.prove_witness: the permutation inputs (16 per row) come
             from pinned host memory, the trace is generated on the device
  host       AirTable.prove: the whole witness comes from pinned host memory
  sumcheck   sumcheck_abc_prove on three device columns (the standalone a*b - c zerocheck)
  noalloc    sumcheck_abc_prove_noalloc, its allocation-free form (at most 2^14 values)
  program    prove_program: an AIR given as a constraint program, witness in host memory
  batch      batch_prove: independent proofs of mixed sizes on a Server's workers
  verify     verify_batch_device: a batch of proofs, some of them broken, with the Merkle paths
             checked on the device
"""
import threading

import numpy as np
import torch

import whirlaway_b200 as wl
from whirlaway_b200 import air_program

P = air_program.P
COLUMNS = 165  # of the Poseidon2 AIR
WORKERS = 8
SERVER_BUDGET = 16 << 30


def listed():
    return [
        # the smallest call: a latency path that must not enter an allocator
        {"name": "sumcheck_noalloc_2p10", "path": "noalloc", "log_n": 10, "skips": 3},
        # a handful of permutations proved on their own: all latency
        {"name": "prove_2p8", "path": "witness", "log_n": 8},
        # the plain single proof of the smallest benchmark configuration
        {"name": "prove_2p12", "path": "witness", "log_n": 12},
        # a mid-size proof with the options of a caller who wants shorter proofs: rate 1/4
        {"name": "prove_2p15_rate4", "path": "witness", "log_n": 15, "log_inv_rate": 2, "univariate_skips": 3},
        # the middle of the served range
        {"name": "prove_2p16", "path": "witness", "log_n": 16},
        # a proving service's request: inputs arrive on the host, the trace is made on the device
        {"name": "inputs_2p18", "path": "inputs", "log_n": 18},
        # a prover whose witness is made elsewhere: 87 MB cross the bus, overlapped with encoding
        {"name": "host_witness_2p17", "path": "host", "log_n": 17},
        # the plain proof at scale, the headline workload
        {"name": "prove_2p20", "path": "witness", "log_n": 20},
        # the sumcheck and folding benchmark at its full size
        {"name": "sumcheck_2p24", "path": "sumcheck", "log_n": 24, "skips": 3},
        # another AIR than the built-in one: transitions of degree 2 with a local constraint
        {"name": "program_mul_2p16", "path": "program", "air": "mul", "log_n": 16},
        # a batch of independent proofs of uneven sizes, as a service gathers them
        {"name": "batch_21", "path": "batch", "proofs": 21, "log_min": 10, "log_max": 15},
        # the other direction: a verifier checks what came in
        {"name": "verify_16", "path": "verify", "proofs": 16, "log_min": 8, "log_max": 12},
    ]


def draw(rng):
    path = rng.choice(["witness", "witness", "witness", "inputs", "host", "sumcheck", "noalloc", "program", "batch",
                       "verify"])
    if path in ("witness", "inputs", "host"):
        rate = rng.choice([1, 1, 2, 3])
        case = {"path": path, "log_n": rng.randint(6, 20 - rate), "log_inv_rate": rate,
                "security_bits": rng.choice([128, 128, 120, 100]), "univariate_skips": rng.choice([4, 4, 3, 2]),
                "rs_domain_initial_reduction": rng.choice([5, 5, 4, 3]), "whir_pow_bits": rng.randint(10, 16)}
        return case
    if path == "sumcheck":
        return {"path": path, "log_n": rng.randint(8, 24), "skips": rng.randint(1, 4)}
    if path == "noalloc":
        return {"path": path, "log_n": rng.randint(8, 14), "skips": rng.randint(1, 4)}
    if path == "program":
        air = rng.choice(["mul", "cubic", "poseidon2"])
        return {"path": path, "air": air, "log_n": rng.randint(8, 15 if air == "poseidon2" else 16),
                "univariate_skips": rng.randint(1, 4)}
    lo = rng.randint(6, 11)
    return {"path": path, "proofs": rng.randint(3, 31) if path == "batch" else rng.randint(9, 15), "log_min": lo,
            "log_max": lo + rng.randint(0, 4 if path == "batch" else 2)}


# ----------------------------------------------------------------------------- state
_lock = threading.Lock()
_kept = {}


def _context():
    """The one context of the program: it owns the stream, the twiddles and the cached buffers."""
    with _lock:
        if "ctx" not in _kept:
            _kept["ctx"] = wl.Context(0)
        return _kept["ctx"]


def _server():
    """The program's server: its workers' contexts live as long as the program."""
    with _lock:
        if "server" not in _kept:
            _kept["server"] = wl.Server(0, workers=WORKERS, hbm_budget_bytes=SERVER_BUDGET)
        return _kept["server"]


def _constants():
    return wl.generate_workload(2, -1, False)[0]


def _settings(case):
    names = ("security_bits", "log_inv_rate", "univariate_skips", "rs_domain_initial_reduction", "whir_pow_bits")
    return wl.AirSettings(**{k: case[k] for k in names if k in case})


def _field(rng, n):
    """n uniform field elements, canonical."""
    return rng.integers(0, P, n, dtype=np.uint32)


def _pinned(n):
    return torch.empty(n, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)


def _mix(case, rng):
    return [int(x) for x in rng.integers(case["log_min"], case["log_max"] + 1, case["proofs"])]


def _program(case, rng, consts):
    """(program, witness) of a constraint-program AIR."""
    log_n, n = case["log_n"], 1 << case["log_n"]
    if case["air"] == "poseidon2":
        w = wl.Witness.generate(_context(), consts, _field(rng, 16 << log_n), log_n)
        wit = w.download()
        w.free()
        return air_program.poseidon2_air_program(consts[:148]), wit
    x, y = [0] * n, [0] * n
    x[0], y[0] = (int(v) for v in rng.integers(1, P, 2))
    if case["air"] == "cubic":  # x' = x^3 + y, y' = x
        for i in range(n - 1):
            x[i + 1] = (x[i] * x[i] * x[i] + y[i]) % P
            y[i + 1] = x[i]
        b = air_program.AirBuilder(2)
        b.assert_zero(b.down(0) - (b.up(0) * b.up(0) * b.up(0) + b.up(1)))
        b.assert_zero(b.down(1) - b.up(0))
        return b.build(), np.array(x + y, dtype=np.uint32)
    for i in range(n - 1):  # x' = x y, y' = y + 1, z = x^2
        x[i + 1] = x[i] * y[i] % P
        y[i + 1] = (y[i] + 1) % P
    b = air_program.AirBuilder(3)
    b.assert_zero(b.down(0) - b.up(0) * b.up(1))
    b.assert_zero(b.down(1) - (b.up(1) + 1))
    b.assert_zero(b.up(2) - b.up(0) * b.up(0))
    return b.build(), np.array(x + y + [v * v % P for v in x], dtype=np.uint32)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    path = case["path"]
    state = {"path": path}
    consts = state["consts"] = _constants()
    if path in ("sumcheck", "noalloc"):
        a, b = (torch.from_numpy(_field(rng, 1 << case["log_n"]).view(np.int32)).cuda() for _ in range(2))
        c = (a.long() * b.long() % P).int()
        state.update(log_n=case["log_n"], skips=case["skips"], p16=consts[148:296], cols=(a, b, c))
        if path == "sumcheck":
            state["ctx"] = _context()
        torch.cuda.synchronize()
        return state
    if path == "batch":
        state["server"] = _server()
        state["jobs"] = [(consts, _field(rng, 16 << n), n) for n in _mix(case, rng)]
        state["words"] = wl.proof_len_bound(wl.AirSettings(), case["log_max"])
        return state
    ctx = state["ctx"] = _context()
    settings = state["settings"] = _settings(case)
    if path == "verify":
        jobs = []
        for n in _mix(case, rng):
            w = wl.Witness.generate(ctx, consts, _field(rng, 16 << n), n)
            proof = wl.AirTable(ctx, consts, n, settings).prove_witness(w)
            w.free()
            if rng.random() < 0.3:  # one word of an opening, a path or a message is wrong
                at = int(rng.integers(0, proof.size))
                proof[at] = (int(proof[at]) + 1) % P
            jobs.append((n, proof))
        state["jobs"] = jobs
        return state
    log_n = state["log_n"] = case["log_n"]
    state["words"] = wl.proof_len_bound(settings, log_n)
    if path == "program":
        state["hash_consts"] = np.ascontiguousarray(consts[148:])
        state["program"], state["witness"] = _program(case, rng, consts)
        return state
    state["table"] = wl.AirTable(ctx, consts, log_n, settings)
    inputs = _field(rng, 16 << log_n)
    if path == "inputs":
        state["inputs"] = _pinned(inputs.size)
        state["inputs"][:] = inputs
        return state
    w = wl.Witness.generate(ctx, consts, inputs, log_n)
    if path == "witness":
        state["witness"] = w
        return state
    state["witness"] = _pinned(COLUMNS << log_n)
    state["witness"][:] = w.download()
    w.free()
    return state


def _record(proof, words):
    """The proof as a record of fixed length with the proof's own length beside it: a proof's
    length varies with the transcript (repeated queries are opened once)."""
    out = np.zeros(words, np.uint32)
    out[: proof.size] = proof
    return out, proof.size


def run(s):
    path = s["path"]
    if path == "witness":
        return _record(s["table"].prove_witness(s["witness"]), s["words"])
    if path == "inputs":
        w = wl.Witness.generate(s["ctx"], s["consts"], s["inputs"], s["log_n"])
        try:
            return _record(s["table"].prove_witness(w), s["words"])
        finally:
            w.free()
    if path == "host":
        return _record(s["table"].prove(s["witness"]), s["words"])
    if path == "sumcheck":
        return wl.sumcheck_abc_prove(s["ctx"], s["p16"], s["log_n"], s["skips"], *s["cols"], device=True)[0]
    if path == "noalloc":
        return wl.sumcheck_abc_prove_noalloc(s["p16"], s["log_n"], s["skips"], *s["cols"])
    if path == "program":
        return _record(wl.prove_program(s["ctx"], s["hash_consts"], s["program"], s["log_n"], s["witness"],
                                        s["settings"]), s["words"])
    if path == "batch":
        return [_record(p, s["words"]) for p in wl.batch_prove(s["server"], s["jobs"])]
    return wl.verify_batch_device(s["ctx"], s["consts"], s["jobs"], s["settings"])


def exact(case, seed):
    """Every output is a sequence of field elements or statuses, whole numbers that have one
    right value each: they are compared as they are."""
    return None


# ----------------------------------------------------------------------------- work
# Field multiplications in the textbook count, two operations each (a product and a sum).
P24_MULTS = 8 * 24 * 2 + 23 * (2 + 24)
P16_MULTS = 8 * 16 * 2 + 20 * (2 + 16)
EF_MULT = 64  # a product in the degree-8 extension
PROOF_BYTES = 4 * 62000


def _prove_work(log_n, rate=1, skips=4, reduction=5, columns=COLUMNS):
    """A proof over a table of `columns` columns: hashing and encoding of the first commitment
    (128-value rows, the columns that are not zero) and of the later ones (each half as long as
    the one before), the zerocheck's points, and one pass of extension-by-base products over
    the witness for the inner sums, the batched column, the two partial evaluations and the
    fold."""
    n = 1 << log_n
    packed = 1 << (columns - 1).bit_length()
    rows0 = (n * packed >> 7) << rate
    rows1 = max(1, (n * packed << rate) >> (4 + reduction))
    mults = rows0 * (8 * P24_MULTS + P16_MULTS) + 2 * rows1 * (8 * P24_MULTS + P16_MULTS)
    mults += rows0 / 2 * max(1, log_n) * 128 * columns / packed + rows1 * max(1, log_n) * 128
    if columns == COLUMNS:
        points = (n >> skips) * (2 * ((1 << skips) - 1))
        mults += points * (148 * (2 + 8) + 148) + 2 * (n >> skips) * 3 * 148 * 3 * EF_MULT
    mults += 5 * 8 * columns * n
    return {"bytes": 4 * columns * n + PROOF_BYTES, "flops": 2 * mults}


def _sumcheck_work(log_n, skips):
    """Three base columns read once; in each round after the skip a fold of three columns and
    two products per point."""
    n = 1 << log_n
    return {"bytes": 12 * n, "flops": 2 * (n * (2 * (1 << skips)) / 2 + n * 24 + 2 * (n >> skips) * 9 * EF_MULT)}


def work(case):
    path = case["path"]
    if path in ("sumcheck", "noalloc"):
        return _sumcheck_work(case["log_n"], case["skips"])
    if path == "program":
        columns = {"mul": 3, "cubic": 2, "poseidon2": COLUMNS}[case["air"]]
        return _prove_work(case["log_n"], skips=case.get("univariate_skips", 4), columns=columns)
    if path in ("batch", "verify"):
        mean = sum(1 << n for n in range(case["log_min"], case["log_max"] + 1)) / (case["log_max"] - case["log_min"] + 1)
        if path == "verify":  # about 130 openings of 8 leaf blocks and a path per proof
            per = 130 * (8 * P24_MULTS + 12 * P16_MULTS)
            return {"bytes": case["proofs"] * PROOF_BYTES, "flops": 2 * per * case["proofs"]}
        one = _prove_work(0)
        return {"bytes": case["proofs"] * (mean * 64 + PROOF_BYTES), "flops": case["proofs"] * mean * one["flops"]}
    w = _prove_work(case["log_n"], case.get("log_inv_rate", 1), case.get("univariate_skips", 4),
                    case.get("rs_domain_initial_reduction", 5))
    if path == "inputs":
        w["bytes"] = 64 * (1 << case["log_n"]) + PROOF_BYTES
    return w
