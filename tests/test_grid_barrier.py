"""The word of the multi-step kernels' grid barrier (csrc/cr_bar.h), compiled as
host code and run through every order in which three CTAs can arrive at a
barrier and poll it: all of them must leave the loop after the same barrier,
the first one at which any of them asked to stop."""
import ctypes as C
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CTAS = 3

SRC = """
#include "cr_bar.h"
extern "C" {
unsigned long long arrival(int k, int stop) { return cr::bar_arrival(k, stop != 0); }
int complete(unsigned long long w, int k, unsigned n) { return cr::bar_complete(w, k, n); }
int stopped(unsigned long long w, int k) { return cr::bar_stopped(w, k); }
}
"""


@pytest.fixture(scope="module")
def bar(tmp_path_factory):
    d = tmp_path_factory.mktemp("bar")
    (d / "bar.cpp").write_text(SRC)
    so = d / "bar.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "cudaring_b200", "csrc"),
                    str(d / "bar.cpp"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.arrival.restype = C.c_ulonglong
    lib.complete.argtypes = [C.c_ulonglong, C.c_int, C.c_uint]
    lib.stopped.argtypes = [C.c_ulonglong, C.c_int]
    return lib


def _outcomes(arrival, complete, stopped, stops, barriers):
    """Every end of the loops: the barrier each CTA left after, or None for a
    state in which some CTA can never pass.  stops: (CTA, barrier) pairs."""
    start = (0, tuple((0, False) for _ in range(CTAS)))  # word; per CTA: its barrier, whether it has arrived
    seen, todo, ends = {start}, [start], set()
    while todo:
        word, ctas = todo.pop()
        nexts = []
        for c, state in enumerate(ctas):
            if isinstance(state, int):
                continue  # left
            k, arrived = state
            if not arrived:
                nexts.append((word + arrival(k, (c, k) in stops), c, (k, True)))
            elif complete(word, k, CTAS):
                leave = stopped(word, k) or k + 1 == barriers
                nexts.append((word, c, k if leave else (k + 1, False)))
        if not nexts:
            ends.add(tuple(s if isinstance(s, int) else None for s in ctas))
        for w, c, s in nexts:
            n = (w, ctas[:c] + (s,) + ctas[c + 1:])
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return ends


def _cases(barriers):
    one = [[(c, k)] for c in range(CTAS) for k in range(barriers)]
    two = [[a, b] for a, b in itertools.combinations([(c, k) for c in range(CTAS) for k in range(barriers)], 2)]
    return [[]] + one + two


def test_every_cta_leaves_after_the_same_barrier(bar):
    barriers = 5
    for stops in _cases(barriers):
        first = min([k for _, k in stops], default=barriers - 1)
        assert _outcomes(bar.arrival, bar.complete, bar.stopped, set(stops), barriers) == {(first,) * CTAS}, stops


def test_one_stop_count_for_all_barriers_would_not_do():
    # the search finds the hang of the former rule: arrivals low, one count of stops above them
    def arrival(k, stop):
        return 1 | (1 << 40 if stop else 0)

    def complete(w, k, n):
        return (w & ((1 << 40) - 1)) >= (k + 1) * n

    ends = _outcomes(arrival, complete, lambda w, k: (w >> 40) != 0, {(0, 1)}, 4)
    assert (1, 1, 1) in ends and any(None in e for e in ends)


def test_counts_do_not_carry(bar):
    # the largest launch: 2 x 64 barriers, every CTA of 65,535 stopping at the last two of them
    ctas, last = 65535, 127
    word = sum(ctas * bar.arrival(k, 0) for k in range(last - 1))
    word += ctas * bar.arrival(last - 1, 1)
    assert bar.complete(word, last - 1, ctas) and not bar.complete(word, last, ctas)
    assert bar.stopped(word, last - 1) and not bar.stopped(word, last)
    word += ctas * bar.arrival(last, 1)
    assert bar.complete(word, last, ctas) and bar.stopped(word, last) and bar.stopped(word, last - 1)
    assert word < 1 << 64
