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


@pytest.mark.parametrize("entry", ["noalloc", "split"])
@pytest.mark.parametrize("degree", range(1, 8))
@pytest.mark.parametrize("modulus,bits", MODULI, ids=[f"{m:#x}"[:12] + f"-{b}" for m, b in MODULI])
def test_a_launch_per_round_matches_c_oracle(modulus, bits, degree, entry):
    """The round kernel alone (sc_prove runs it for the largest rounds only): every register class,
    with and without a fold, and rounds of 4096 pairs that take g(1) from the claim -- on one rank,
    and from the shares of two."""
    from test_gpu_split import _emulate
    from test_zz_no_alloc import _noalloc

    spec = field_for_modulus(modulus, bits)
    expr = expression(degree, 300 + degree)
    terms, k = O.indexed_terms(expr)
    n = 14 if entry == "noalloc" else 15  # two ranks: 2^14 entries each
    tables = api.generate_tables(spec, k, n, [0] * k, degree)
    want = C.prove_seeded(terms, k, spec.modulus, spec.limbs, n, [0] * k, degree)
    if entry == "noalloc":
        ctx = api.get_context(tables.device)
        ce = api.CompiledExpression(api.encode_expression(expr), spec.modulus)
        rc, *got = _noalloc(ctx, api.get_device_field(spec, ctx.device), ce, n, tables, "sha3", spec.limbs, degree, k)
        assert rc == api._lib.SC_OK, api._lib.last_error()
        results = [got]
    else:
        results = [(p.round_polys_mont, p.challenges_mont, p.finals_mont, p.claim0_mont, p.checksum)
                   for p in _emulate(tables, expr, spec, n, 2)]
    for polys, chals, finals, claim0, checksum in results:
        assert np.array_equal(polys, want["round_polys"])
        assert np.array_equal(chals, want["challenges"])
        assert np.array_equal(finals, want["finals"])
        assert np.array_equal(claim0, want["claim0"])
        assert checksum == want["checksum"]


@pytest.mark.parametrize("degree", [2, 4, 7])
@pytest.mark.parametrize("modulus,bits,n", [(m, b, 18 if b == 256 else 16) for m, b in MODULI[:4] + MODULI[-2:]])
def test_large_rounds_then_parts_and_a_tail_match_c_oracle(modulus, bits, n, degree):
    check(expression(degree, 500 + degree), field_for_modulus(modulus, bits), n, seed=n + degree)


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
