"""A served prover after a failing call (GPU): every request it holds ends with the error, none is
left waiting, and what they held -- staging slots, budget, device blocks -- is free for the next.

The failures are made on the host: a library loaded in front of the prover's stands in for the
call that fails (table generation at an admission, a tick's launch) and returns an error code
without calling on; every other call goes through. Each test is a child process of its own.
"""

from __future__ import annotations

import re
import subprocess
import sys
from pathlib import Path

import pytest

from zkduel_b200 import _lib

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a GPU", allow_module_level=True)

ROOT = Path(__file__).resolve().parents[1]

SHIM = r"""
#include <stdint.h>
#include <unistd.h>
typedef int (*tables_fn)(void*, const void*, int, int, const int32_t*, uint64_t, uint32_t*);
typedef int (*launch_fn)(int, int, int, const void*, unsigned, int, size_t, void*, const void*, _Bool);
static tables_fn real_tables;
static launch_fn real_launch;
volatile int fail_tables, fail_launches, pass_launches, hold, held;
void set_real(void* tables, void* launch) { real_tables = (tables_fn)tables; real_launch = (launch_fn)launch; }
void set_fail(int tables, int launches, int after) { fail_tables = tables; fail_launches = launches; pass_launches = after; }
void set_hold(int on) { hold = on; }
int is_held(void) { return held; }
int sc_tables_generate(void* ctx, const void* f, int k, int n, const int32_t* kinds, uint64_t seed, uint32_t* out) {
  if (fail_tables > 0) { --fail_tables; return 3; }
  return real_tables(ctx, f, k, n, kinds, seed, out);
}
int launch(int L, int K, int d, const void* f, unsigned g, int t, size_t s, void* st, const void* T, _Bool a) __asm__("LAUNCH");
int launch(int L, int K, int d, const void* f, unsigned g, int t, size_t s, void* st, const void* T, _Bool a) {
  for (int i = 0; hold && i < 200000; ++i) { held = 1; usleep(100); }
  held = 0;
  if (fail_launches > 0 && pass_launches-- <= 0) { --fail_launches; return 3; }
  return real_launch(L, K, d, f, g, t, s, st, T, a);
}
"""

CHILD = r"""
import ctypes, os, sys, time
sys.path.insert(0, sys.argv[1] + "/sumcheck-triton_b200")
shim = ctypes.CDLL(sys.argv[2], mode=ctypes.RTLD_GLOBAL)  # in front of the library's own symbols
import numpy as np
import torch
from zkduel_b200 import _lib, api
from zkduel_b200.fields import get_field
from zkduel_b200.serve import ProofServer
lib = _lib.load()
real = [ctypes.cast(getattr(lib, n), ctypes.c_void_p) for n in ("sc_tables_generate", sys.argv[3])]
shim.set_real(*real)
spec, expr = get_field(128), ((1, ("a", "b")), (2, ("c",)))

def check(srv, rid, n, seed):
    t = api.generate_tables(spec, 3, n, [0] * 3, seed)
    a, b = srv.result(rid), api.prove_device(t, expr, spec, n)
    assert np.array_equal(a.round_polys_mont, b.round_polys_mont) and np.array_equal(a.finals_mont, b.finals_mont)

def fails(srv, rid):
    try:
        srv.wait(rid, timeout_ms=10_000)
    except TimeoutError:
        raise
    except _lib.SumcheckError:
        return
    raise AssertionError("the request did not fail")

def admissions(n):
    # two staging slots and a budget of one and a half requests: a leak of either is felt at once
    srv = ProofServer(spec, max_inflight=2)
    srv = ProofServer(spec, max_inflight=2, budget_bytes=srv.footprint(expr, n) * 3 // 2)
    for i in range(3):
        shim.set_fail(1, 0, 0)
        fails(srv, srv.submit(expr, n, i))
    rid = srv.submit(expr, n, 9)
    srv.wait(rid, timeout_ms=10_000)
    check(srv, rid, n, 9)
    st = srv.stats()
    assert (st["failed"], st["completed"]) == (3, 1), st
    srv.close()

def ticks(with_suspension):
    srv = ProofServer(spec, max_inflight=4, threads=32)
    shim.set_hold(1)
    ids = [srv.submit(expr, 12, i) for i in range(2 if with_suspension else 1)]
    while not shim.is_held():  # the worker is in the launch of a tick
        time.sleep(0.001)
    if with_suspension:  # leaves with the next tick, whose launch (the other request's) fails
        srv.suspend(ids[0])
    shim.set_fail(0, 1, 1 if with_suspension else 0)
    shim.set_hold(0)
    for rid in ids:
        fails(srv, rid)
    rid = srv.submit(expr, 12, 9)
    srv.wait(rid, timeout_ms=10_000)
    check(srv, rid, 12, 9)
    srv.close()

{"small": lambda: admissions(9), "large": lambda: admissions(19), "tick": lambda: ticks(False),
 "suspended": lambda: ticks(True)}[sys.argv[4]]()
print("CHILD OK", flush=True)
os._exit(0)
"""


@pytest.mark.parametrize("case", ["small", "large", "tick", "suspended"])
def test_a_failing_call_ends_every_request_and_leaves_the_server_usable(case, tmp_path):
    names = subprocess.run(["nm", "-D", str(_lib.LIB_PATH)], capture_output=True, text=True, check=True).stdout
    launch = re.search(r"T (_ZN7sc_host19batch_kernel_launchE\w+)", names)[1]
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM.replace("LAUNCH", launch))
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(lib)], check=True)
    child = tmp_path / "child.py"
    child.write_text(CHILD)
    r = subprocess.run([sys.executable, str(child), str(ROOT), str(lib), launch, case], capture_output=True, text=True,
                       timeout=180)
    assert r.returncode == 0 and "CHILD OK" in r.stdout, r.stdout[-1000:] + r.stderr[-3000:]
