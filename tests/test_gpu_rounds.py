"""Whole proofs over the range of the round kernels, bit-exact against the C oracle (GPU).

Every limb count, every degree (one to three hash blocks a round, every register class), sizes
from one pair to rounds of more blocks than the grid's sums have copies, and moduli at the ends
of what a limb count holds: tiny, a little below half of it, and the largest the modulus guard lets through.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import c_oracle as C
from oracle import oracle as O
from zkduel_b200 import api
from zkduel_b200.fields import field_for_modulus, get_field

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a GPU", allow_module_level=True)

# (modulus, bits): the configured fields, then the ends of each limb count's range
MODULI = [(get_field(b).modulus, b) for b in (32, 64, 128, 256)] + [
    (65537, 32), ((1 << 61) - 1, 64), (97, 64), ((1 << 128) - (1 << 96) - 11, 128), ((1 << 89) - 1, 128),
    (10007, 256), ((1 << 255) - 19, 256), ((1 << 256) - (1 << 224) - 53, 256),
]


def expression(degree, seed):
    """A sum of products of that degree: one full term, one shorter, one of repeated factors."""
    rng = np.random.default_rng(seed)
    names = [f"t{i}" for i in range(max(2, degree))]
    terms = [(1, names[:degree])]
    if degree > 1:
        terms.append((-3, [names[i] for i in rng.permutation(len(names))[: degree - 1]]))
        terms.append((5, [names[0]] * int(rng.integers(1, degree + 1))))
    return terms


def check(expr, spec, n, seed):
    terms, k = O.indexed_terms(expr)
    kinds = [api._lib.SC_TABLE_UNIFORM] * k
    tables = api.generate_tables(spec, k, n, kinds, seed)
    got = api.prove_device(tables, expr, spec, n)
    want = C.prove_seeded(terms, k, spec.modulus, spec.limbs, n, [0] * k, seed)
    assert np.array_equal(got.round_polys_mont, want["round_polys"])
    assert np.array_equal(got.challenges_mont, want["challenges"])
    assert np.array_equal(got.finals_mont, want["finals"])
    assert np.array_equal(got.claim0_mont, want["claim0"])
    assert got.checksum == want["checksum"]


@pytest.mark.parametrize("degree", range(1, 8))
@pytest.mark.parametrize("modulus,bits", MODULI, ids=[f"{m:#x}"[:12] + f"-{b}" for m, b in MODULI])
def test_every_degree_matches_c_oracle(modulus, bits, degree):
    spec = field_for_modulus(modulus, bits)
    for n in (1, 2, 6, 9, 13):
        check(expression(degree, 100 * degree + n), spec, n, seed=degree + n)


@pytest.mark.parametrize("bits", [32, 64, 128, 256])
@pytest.mark.parametrize("n", [15, 17])
def test_many_blocks_match_c_oracle(bits, n):
    check(expression(3, n), get_field(bits), n, seed=n)


def test_tick_times_follow_each_other():
    from zkduel_b200.batch import BatchProver

    for bits, n in ((32, 1), (64, 5), (256, 9)):
        spec = get_field(bits)
        expr = ((1, ("a", "b")), (3, ("c",)))
        bp = BatchProver([(expr, bits, n, api.generate_tables(spec, 3, n, [0] * 3, 7))])
        with pytest.raises(Exception):
            bp.tick_times()  # not run yet
        for _ in range(2):
            bp.run()
            (c,) = bp.tick_times()
            assert len(c["ms"]) == n and c["start"][0] == 0.0
            assert all(0 < b - a < 1e3 for a, b in zip(c["start"], c["end"]))
            assert all(nxt >= end for end, nxt in zip(c["end"], c["start"][1:]))
