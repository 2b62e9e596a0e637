"""Pinned host blocks are page-locked once: uploads of batches and copies of
their records, large and small in turn, go on with the blocks of the first
round.  A preloaded cudaHostAlloc counts the calls."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_COUNT = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int calls;
int pinned_calls(void) { return calls; }
int cudaHostAlloc(void** p, size_t n, unsigned flags) {
  static int (*next)(void**, size_t, unsigned);
  void* rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);  /* loaded by the library, not globally */
  if (rt && !next) next = (int (*)(void**, size_t, unsigned))dlsym(rt, "cudaHostAlloc");
  if (!next) return 999;
  ++calls;
  return next(p, n, flags);
}
"""

_ROUNDS = """
import ctypes, sys
import poker_solver_rust_b200 as ps
from tests import spots
count = ctypes.CDLL(sys.argv[1]).pinned_calls
def batch(n):
    sp = spots.datagen_spots(n, seed=3)
    return [spots.card_config(r, b) for r, b, _ in sp], [t for _, _, t in sp]
sizes = [batch(1200), batch(250)]  # records of about 41 and 8.6 MB: more pieces than one thread's, and few
calls = []
for _ in range(6):
    for cards, trees in sizes:
        b = ps.BatchSolver(cards, trees)
        b.solve(1, [0.0] * len(cards))
        b.records()
        del b
    calls.append(count())
print("CALLS", *calls)
"""


def test_blocks_are_locked_once(tmp_path):
    src, lib = tmp_path / "count.c", tmp_path / "count.so"
    src.write_text(_COUNT)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", _ROUNDS, str(lib)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(lib)))
    assert r.returncode == 0, r.stderr
    calls = [int(x) for x in r.stdout.split("CALLS")[1].split()]
    assert calls[0] > 0 and calls[-1] == calls[1], calls
