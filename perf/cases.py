"""The work that programs built on zkduel_b200 have it do, as timed cases.

A case names an entry point of the package (``entry``) and the sizes of one call:

prove   ``api.prove_device``: one proof over tables resident on the GPU.
seeded  ``api.prove``: (expression, field width, num_vars, seed) -> proof, tables generated
        on the GPU inside the call.
host    ``api.sumcheck``: canonical host tables and explicit challenges in, claim and round
        polynomials out (the drop-in call).
batch   ``batch.BatchProver``: many proofs of mixed sizes, fields and degrees over resident
        tables, run and read back.
ingest  ``batch.HostBatchProver``: the same from tables in pinned host memory.
serve   ``serve.ProofServer``: a burst of requests submitted, awaited and read back.

Everything returned is whole numbers (Montgomery limbs, checksums, canonical values).
"""

from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "sumcheck-triton_b200"))

from zkduel_b200 import _lib, api  # noqa: E402
from zkduel_b200.batch import BatchProver, HostBatchProver  # noqa: E402
from zkduel_b200.expression import encode_expression  # noqa: E402
from zkduel_b200.fields import get_field  # noqa: E402
from zkduel_b200.serve import ProofServer  # noqa: E402
from zkduel_b200.streams import batched_stream, served_stream  # noqa: E402
from zkduel_b200.workloads import WORKLOADS  # noqa: E402

# selector tables of the zerocheck gates are 0/1, every other table is uniform
SELECTORS = {"qM", "qL", "qR", "qO", "q1", "q2", "q3", "q4", "qM1", "qM2", "qH1", "qH2", "qH3", "qH4", "qECC"}

# registry expressions that drawn single proofs use: degrees 1 to 7, 1 to 17 terms, with and
# without coefficients and repeated factors
PLAIN_WORKLOADS = [
    "poly_ab", "poly_ab_plus_c", "poly_abc", "poly_aabbc", "poly_abcg_plus_deg", "cubic_plus_quad", "opencheck",
    "vanilla_zerocheck_hp", "vanilla_permcheck_hp", "jellyfish_zerocheck_hp", "jellyfish_permcheck_hp",
    "verifiable_asics", "spartan_1", "spartan_2", "witness_id_point_1", "incomplete_addition_1",
    "complete_addition_3", "complete_addition_7",
]


def listed():
    return [
        # one small proof: a call is all launches and latency
        {"name": "ab_32bit_n8", "entry": "prove", "workload": "poly_ab", "bits": 32, "n": 8},
        # the small plain configuration: two tables of 2^16 entries
        {"name": "ab_32bit_n16", "entry": "prove", "workload": "poly_ab", "bits": 32, "n": 16},
        # the same gate as the large plain configuration at the size of a small circuit
        {"name": "zerocheck_64bit_n13", "entry": "prove", "workload": "vanilla_zerocheck_hp", "bits": 64, "n": 13},
        # the plain 64-bit configuration: nine tables of 2^24 entries, 1.2 GB
        {"name": "zerocheck_64bit_n24", "entry": "prove", "workload": "vanilla_zerocheck_hp", "bits": 64, "n": 24},
        # a permutation check (coefficients, ten tables, degree 5) of an ordinary circuit
        {"name": "permcheck_64bit_n19", "entry": "prove", "workload": "vanilla_permcheck_hp", "bits": 64, "n": 19},
        # the plain 256-bit configuration: six tables of 2^22 entries
        {"name": "abcg_256bit_n22", "entry": "prove", "workload": "poly_abcg_plus_deg", "bits": 256, "n": 22},
        # a custom gate of many low-degree terms over the 256-bit field
        {"name": "addition_256bit_n15", "entry": "prove", "workload": "incomplete_addition_1", "bits": 256, "n": 15},
        # the seeded call over the 128-bit field, with repeated factors
        {"name": "seeded_128bit_n17", "entry": "seeded", "workload": "poly_aabbc", "bits": 128, "n": 17},
        # the drop-in call on host tables
        {"name": "host_64bit_n12", "entry": "host", "workload": "spartan_1", "bits": 64, "n": 12},
        # the mixed stream: 64- and 256-bit proofs, n 10 to 20, degree 2 to 6
        {"name": "batch_64", "entry": "batch", "count": 64, "n_min": 10, "n_max": 20},
        # the same proofs' smaller half arriving from host memory
        {"name": "ingest_24", "entry": "ingest", "count": 24, "n_min": 10, "n_max": 17},
        # a burst of served requests over 2^127 - 1, degree 3 to 7
        {"name": "serve_40", "entry": "serve", "count": 40, "n_min": 12, "n_max": 20},
    ]


def draw(rng):
    entry = rng.choices(["prove", "seeded", "host", "batch", "ingest", "serve"], [8, 2, 1, 3, 1, 2])[0]
    if entry in ("prove", "seeded"):
        # a registry expression, or one of the mixed stream's random sums of products
        workload = rng.choice(PLAIN_WORKLOADS) if rng.random() < 0.5 else "mixed_%d" % rng.randrange(1, 100000)
        bits = rng.choice([32, 64, 128, 256])
        limbs = bits // 32
        # tables of at most 400 MB, and no more products than the largest listed case
        expr = _expression(workload)
        top = int(math.log2(4e8 / (4 * limbs * encode_expression(expr).num_vars)))
        while top > 7 and _products(expr, top) * limbs * limbs > 8e9:
            top -= 1
        # the logarithm of the table size is uniform
        return {"entry": entry, "workload": workload, "bits": bits, "n": rng.randint(6, min(top, 24))}
    if entry == "host":
        return {"entry": "host", "workload": rng.choice(["spartan_1", "poly_abc", "verifiable_asics"]),
                "bits": rng.choice([32, 64]), "n": rng.randint(6, 13)}
    count = int(round(math.exp(rng.uniform(math.log(4), math.log(64 if entry == "batch" else 40)))))
    lo = rng.randint(8, 12)
    return {"entry": entry, "count": count, "n_min": lo, "n_max": rng.randint(lo + 2, 18 if entry == "batch" else 17)}


def _expression(workload):
    if workload.startswith("mixed_"):
        return batched_stream(1, seed=int(workload[6:]))[0].expression
    return WORKLOADS[workload]


def _products(expression, n):
    enc = encode_expression(expression)
    muls = sum(max(0, length - 1) for length in enc.term_lens)
    return (enc.degree + 1) * muls * (1 << n) + 2 * enc.num_vars * (1 << n)


def _kinds(expression):
    names = encode_expression(expression).var_names
    return [_lib.SC_TABLE_BERNOULLI if v in SELECTORS else _lib.SC_TABLE_UNIFORM for v in names]


def _stream(case):
    """(expression, field width, num_vars) of every proof of a batch or burst: the kinds of the
    package's streams, cut to the case's range of sizes. Shapes depend on the case alone."""
    count, lo, hi = case["count"], case["n_min"], case["n_max"]
    sizes = random.Random(count * 1000 + lo * 50 + hi)
    if case["entry"] == "serve":
        reqs = served_stream(count, seed=1)
        return [(r.spec.expression, 128,
                 int(round(math.exp(sizes.uniform(math.log(lo), math.log(hi)))))) for r in reqs]
    return [(s.expression, s.bit_width, sizes.randint(lo, hi)) for s in batched_stream(count, seed=1)]


def prepare(case, seed):
    entry = case["entry"]
    if entry in ("prove", "seeded", "host"):
        expr = _expression(case["workload"])
        spec, n = get_field(case["bits"]), case["n"]
        enc = encode_expression(expr)
        if entry == "seeded":
            return {"entry": entry, "expr": expr, "bits": case["bits"], "n": n, "seed": seed,
                    "kinds": ["bernoulli" if v in SELECTORS else "uniform" for v in enc.var_names]}
        if entry == "prove":
            return {"entry": entry, "expr": api.CompiledExpression(enc, spec.modulus), "spec": spec, "n": n,
                    "tables": api.generate_tables(spec, enc.num_vars, n, _kinds(expr), seed)}
        rng = np.random.default_rng(seed)
        return {"entry": entry, "expr": expr, "q": spec.modulus, "bits": case["bits"], "n": n,
                "tables": {v: rng.integers(0, spec.modulus, 1 << n, dtype=np.uint64) for v in enc.var_names},
                "challenges": [int(x) for x in rng.integers(0, spec.modulus, n, dtype=np.uint64)]}
    proofs = _stream(case)
    if entry == "serve":
        server = ProofServer(128, budget_bytes=4 * 10**9)
        server.reserve(2 * 10**9)
        rng = random.Random(seed)
        return {"entry": entry, "server": server,
                "requests": [(api.CompiledExpression(encode_expression(e), server.spec.modulus), n, rng.getrandbits(63))
                             for e, _b, n in proofs]}
    items, rng = [], random.Random(seed)
    for e, bits, n in proofs:
        spec = get_field(bits)
        ce = api.CompiledExpression(encode_expression(e), spec.modulus)
        t = api.generate_tables(spec, ce.num_vars, n, [_lib.SC_TABLE_UNIFORM] * ce.num_vars, rng.getrandbits(63))
        items.append((ce, bits, n, t))
    if entry == "batch":
        return {"entry": entry, "prover": BatchProver(items)}
    host = []
    for _e, bits, _n, t in items:
        limbs = api.download_tables(t, get_field(bits)).view(np.int32)
        h = torch.empty(limbs.shape, dtype=torch.int32, pin_memory=True)
        h.copy_(torch.from_numpy(limbs))
        host.append(h)
    return {"entry": entry, "prover": HostBatchProver([(e, b, n) for e, b, n, _t in items], host, chunks=4)}


def _outputs(proofs):
    """Every output of the proofs, each kind in one flat array."""
    return {
        "round_polys": np.concatenate([p.round_polys_mont.ravel() for p in proofs]),
        "challenges": np.concatenate([p.challenges_mont.ravel() for p in proofs]),
        "finals": np.concatenate([p.finals_mont.ravel() for p in proofs]),
        "claims": np.concatenate([p.claim0_mont for p in proofs]),
        "checksums": np.array([p.checksum for p in proofs], dtype=np.uint64),
    }


def run(state):
    entry = state["entry"]
    if entry == "prove":
        return _outputs([api.prove_device(state["tables"], state["expr"], state["spec"], state["n"])])
    if entry == "seeded":
        return _outputs([api.prove(state["expr"], state["bits"], state["n"], state["seed"], table_kinds=state["kinds"])])
    if entry == "host":
        claim, evals = api.sumcheck(state["tables"], q=state["q"], expression=state["expr"],
                                    challenges=state["challenges"], num_rounds=state["n"], bit_width=state["bits"])
        return {"claim": np.array([claim], dtype=np.uint64), "evals": evals.astype(np.uint64)}
    if entry == "batch":
        state["prover"].run()
        return _outputs(state["prover"].results())
    if entry == "ingest":
        return _outputs(state["prover"].run())
    server = state["server"]
    ids = [server.submit(e, n, s) for e, n, s in state["requests"]]
    for rid in ids:
        server.wait(rid)
    proofs = [server.result(rid) for rid in ids]
    for rid in ids:
        server.release(rid)
    return _outputs(proofs)


def _proof_work(expression, bits, n):
    """Bytes: every table read once, the outputs written once. Operations: two for every 32-bit
    multiply-add of the proof's Montgomery products (d + 1 points of every pair of every round,
    two products per table and folded pair), 2 L^2 + L of them a product."""
    enc = encode_expression(expression)
    limbs, size, d = bits // 32, 1 << n, enc.degree
    per_point = sum(max(0, length - 1) for length in enc.term_lens)
    products = (size - 1) * (d + 1) * per_point + enc.num_vars * (size - 2)
    data = 4 * limbs * (enc.num_vars * size + n * (d + 2) + enc.num_vars + 2)
    return data, 2 * products * (2 * limbs * limbs + limbs)


def work(case):
    if case["entry"] in ("prove", "seeded", "host"):
        proofs = [(_expression(case["workload"]), case["bits"], case["n"])]
    else:
        proofs = _stream(case)
    data, ops = zip(*(_proof_work(*p) for p in proofs))
    return {"bytes": sum(data), "flops": sum(ops)}


def exact(case, seed):
    """Outputs are whole numbers, equal bit for bit or wrong: there is nothing to be near to."""
    return None
