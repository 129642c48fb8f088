"""The inline-PTX arithmetic of csrc/field_m127.cuh (any representatives of residues mod
2^127 - 1 below 2^128), csrc/field_gold_acc.cuh (Goldilocks sums of products reduced once) and
csrc/field_bls_fold.cuh (folds over the BLS12-381 scalar field from a table of the challenge), run on the CPU statement by statement against big integers: random operands and the edges of
the representations (0, p, 2^127, 2^128 - 1, full words, and their neighbours)."""

from __future__ import annotations

import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "sumcheck-triton_b200" / "csrc"
M32 = (1 << 32) - 1
P = (1 << 127) - 1
EDGES = [0, 1, 2, P - 1, P, P + 1, P + 2, (1 << 127) + 5, (1 << 128) - 3, (1 << 128) - 2, (1 << 128) - 1, 2 * P, 2 * P + 1]


def _programs():
    out = {}
    for header in ("field_m127.cuh", "field_gold_acc.cuh", "field_bls_fold.cuh"):
        for name, body in re.findall(r"void ((?:m127|gold|bls)_\w+)\((.*?)\n\}\n", (CSRC / header).read_text(), re.S):
            asm = body.split("asm(")[1]
            text = "".join(re.findall(r'"((?:[^"\\]|\\.)*)"', re.split(r'\n      : "[=+]', asm)[0]))
            lines = [ln.strip().rstrip(";") for ln in text.replace("\\n", "\n").replace("\\t", "").split("\n")]
            outs = len(re.findall(r'"(?:=&|\+)r"', asm))
            tied = re.findall(r'"\+r"\((\w+)\[(\d)\]\)', asm)
            ins = tied + re.findall(r'"r"\(([\w.]+)(?:\[(\d)\])?\)', asm)
            out[name] = (bool(tied), [ln for ln in lines if ln and ln not in "{}" and not ln.startswith(".reg")], outs, ins)
    return out


PROGRAMS = _programs()
GOLD = (1 << 64) - (1 << 32) + 1
GOLD_K = {"k.one": 1, "k.zero": 0, "k.eps": M32}


def run(name, **operands):
    """The value (its words low to high) the statement leaves in its outputs."""
    tied, lines, outs, ins = PROGRAMS[name]
    operands.update(GOLD_K)
    first = 0 if tied else outs  # read-write operands come first and are inputs too
    regs = {f"%{first + i}": operands[v] >> (32 * int(k or 0)) & M32 for i, (v, k) in enumerate(ins)}
    flag = family = None
    val = lambda x: regs[x] if x in regs else int(x, 0) & M32  # noqa: E731
    for ln in lines:
        op, rest = ln.split(None, 1)
        args = [a.strip() for a in rest.split(",")]
        kind, d, a = op.split(".")[0], args[0], [val(x) for x in args[1:]]
        if kind in ("addc", "madc", "subc"):
            assert family == ("sub" if kind == "subc" else "add"), f"{name}: {ln} reads the other family's flag"
        cin = flag if kind in ("addc", "madc", "subc") else 0
        if kind == "mov":
            s = a[0]
        elif kind in ("mul", "mad", "madc"):
            prod = a[0] * a[1]
            s = (prod & M32 if ".lo" in op else prod >> 32) + (a[2] + cin if kind != "mul" else 0)
        elif kind in ("add", "addc"):
            s = a[0] + a[1] + cin
        elif kind in ("sub", "subc"):
            s = a[0] - a[1] - cin
        elif kind == "and":
            s = a[0] & a[1]
        elif kind == "shl":
            s = a[0] << a[1] & M32
        elif kind == "shr":
            s = a[0] >> a[1]
        elif kind == "shf":
            s = ((a[1] << 32 | a[0]) >> a[2]) & M32
        else:
            raise ValueError(ln)
        if ".cc" in op:
            flag, family = int(s < 0 or s > M32), "sub" if kind.startswith("sub") else "add"
        regs[d] = s & M32
    return sum(regs[f"%{k}"] << (32 * k) for k in range(outs))


def pairs(seed, count):
    rng = random.Random(seed)
    out = [(a, b) for a in EDGES for b in EDGES]
    for _ in range(count):
        a, b = rng.getrandbits(128), rng.getrandbits(128)
        if rng.random() < 0.3:
            a = (1 << 128) - 1 - rng.getrandbits(rng.randrange(1, 100))
        if rng.random() < 0.3:
            b = rng.getrandbits(rng.randrange(1, 128))
        out.append((a, b))
    return out


@pytest.mark.parametrize("name,want", [
    ("m127_mul_lazy", lambda a, b: a * b * pow(1 << 128, -1, P)),
    ("m127_add_lazy", lambda a, b: a + b),
    ("m127_sub_lazy", lambda a, b: a - b),
])
def test_lazy_forms_match_big_integers(name, want):
    for a, b in pairs(7, 3000):
        got = run(name, x=a, y=b) if name == "m127_mul_lazy" else run(name, a=a, b=b)
        assert got % P == want(a, b) % P, (hex(a), hex(b))


def test_canonical_form():
    for a, b in pairs(9, 1500):
        for x in (a, b):
            assert run("m127_canon", a=x) == x % P, hex(x)


def test_bls_folds_from_a_table():
    p = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
    rng = random.Random(4)
    edge = lambda: rng.choice([0, 1, p - 1, p - 2, (1 << 254) - 1, rng.randrange(p), rng.randrange(p)])  # noqa: E731
    for _ in range(400):
        r, x0, x = edge(), edge(), edge()
        table = [r * (1 << (32 * i + 64)) % p for i in range(8)]
        e, o = x0 << 64, 0
        for i in range(8):
            eo = run("bls_fold_row", e=e, o=o, x=x >> (32 * i) & M32, c=table[i])
            e, o = eo & ((1 << 320) - 1), eo >> 320
        assert e + (o << 32) == (x0 << 64) + sum((x >> (32 * i) & M32) * table[i] for i in range(8))
        got = run("bls_fold_end", e=e, o=o, p=p)
        assert got % p == (x0 + r * x) % p and got < x0 + p + (p >> 28)


def test_goldilocks_sums_of_products():
    rng = random.Random(3)
    edges = [0, 1, M32, 1 << 32, GOLD - 1, GOLD, GOLD + 1, (1 << 64) - 1, (1 << 64) - (1 << 32), (1 << 63)]
    word = lambda: rng.choice(edges) if rng.random() < 0.5 else rng.getrandbits(64)  # noqa: E731
    r_inv = pow(1 << 64, -1, GOLD)
    for _ in range(4000):
        x, y = word(), word()
        t = run("gold_acc_first", x=x, y=y)
        assert t == x * y
        want = x * y
        for _ in range(rng.randrange(6)):
            x, y = word(), word()
            t = run("gold_acc_mul", t=t, x=x, y=y)
            want += x * y
        if rng.random() < 0.5:
            x = word()
            t = run("gold_acc_add", t=t, x=x)
            want += x << 64
        assert t == want
        # the carries of up to 2^31 products above 128 bits
        t += rng.choice([0, 0, rng.getrandbits(31), (1 << 31) - 1 - (t >> 128)]) << 128
        t = min(t, ((1 << 31) << 128) - 1)
        assert run("gold_acc_reduce", t=t) % GOLD == t * r_inv % GOLD, hex(t)
    for a in edges[:6]:
        assert run("gold_neg", a=a) == GOLD - a if a <= GOLD else True
