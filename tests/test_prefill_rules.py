"""Rules of the tcgen05 prompt attention (``csrc/prefill_rules.h``), compiled as plain C++: the order of the waits on the
barrier of O += P V, walked through in every interleaving."""

import ctypes
import itertools
import os
import random
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mini_infer_b200", "csrc")
SOURCE = """
#include "prefill_rules.h"
using namespace mi;
extern "C" int follows_product(int j, int n, int rescale) { return pt::follows_product(j, n, rescale != 0); }
extern "C" int query_order(int64_t longest, int64_t total, int heads, int requests, int dk, int bounded) {
    return pt::query_order(longest, total, heads, requests, dk, bounded != 0);
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    folder = tmp_path_factory.mktemp("rules")
    (folder / "rules.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror", "-I", CSRC, str(folder / "rules.cpp"), "-o",
                    str(folder / "rules.so")], check=True)
    lib = ctypes.CDLL(str(folder / "rules.so"))
    lib.query_order.argtypes = [ctypes.c_int64, ctypes.c_int64] + [ctypes.c_int] * 4
    return lib


def program(n, rescales, follows):
    """What a softmax warp does: ("tile", j) S of tile j is there; ("wait", k) on phase k's parity; ("give", j) P of tile j."""
    out = []
    for j in range(n):
        out.append(("tile", j))
        if follows(j, n, rescales[j]):
            out.append(("wait", j - 1))
        out.append(("give", j))
    return out + [("wait", n - 1)]


def lost_or_early(programs, n):
    """Every interleaving of the warps and the products: a wait that passes before its phase is complete, or a state in
    which nobody can go on before all have ended.  State: each warp's place and the number of completed products."""
    seen, stack = set(), [((0,) * len(programs), 0)]
    while stack:
        state = stack.pop()
        if state in seen:
            continue
        seen.add(state)
        at, done = state
        given = [sum(kind == "give" for kind, _ in p[:i]) for p, i in zip(programs, at)]
        nxt = [(at, done + 1)] if done < min(given) else []          # product `done` has every warp's P
        for w, (p, i) in enumerate(zip(programs, at)):
            if i == len(p):
                continue
            kind, k = p[i]
            if kind == "tile" and done < k - 1:                      # S of tile k is issued after product k - 2
                continue
            if kind == "wait":
                if done & 1 == k & 1:                                # the current phase has the parity waited for
                    continue
                if done <= k:
                    return f"warp {w} passes phase {k} after {done} products"
            nxt.append((at[:w] + (i + 1,) + at[w + 1:], done))
        if not nxt and any(i < len(p) for p, i in zip(programs, at)):
            return f"nobody goes on at {state}"
        stack.extend(nxt)
    return None


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_no_wait_on_a_product_is_lost(rules, n):
    follows = lambda j, n, r: bool(rules.follows_product(j, n, int(r)))
    for a, b in itertools.product(itertools.product([False, True], repeat=n), repeat=2):
        programs = [program(n, a, follows), program(n, b, follows)]
        assert lost_or_early(programs, n) is None, (a, b)


def test_the_walk_finds_a_wait_behind_the_last_hand_over():
    late = lambda rescales: program(3, rescales, lambda j, n, r: j > 0 and r)[:-1] + [("wait", 1), ("wait", 2)]
    assert lost_or_early([late([False] * 3), late([False] * 3)], 3)
    none = lambda j, n, r: False
    assert lost_or_early([program(3, [False] * 3, none)] * 2, 3)


def test_a_whole_warps_wait_is_agreed_upon():
    """Lanes may give a wait up one by one (a limit each), and what follows is for whole warps: every wait that is not one
    lane's alone is followed by a vote before anything else looks at its outcome."""
    source = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "attention_prefill_tc.cu")).read())
    statements = [re.sub(r"\s+", " ", s).strip() for s in source.split(";")]
    waits = [i for i, s in enumerate(statements)
             if re.search(r"\bok = .*(mbar_wait|k_there)\(", s) and "if (lane == 0) ok =" not in s]
    assert len(waits) >= 7
    for i in waits:
        if "ok = __all_sync(0xffffffffu, k_there(" in statements[i]:         # the vote is around the wait
            continue
        assert re.match(r"ok = (together = )?(__all_sync|pair_and)\(", statements[i + 1]), (statements[i], statements[i + 1])


SINGLE, APART, NEIGHBOURS = 0, 1, 2


@pytest.mark.parametrize("lengths,heads,order", [
    ([2048], 16, APART), ([2048], 8, SINGLE), ([8192], 16, NEIGHBOURS), ([1000] * 3, 16, NEIGHBOURS),
    ([1000, 100, 100], 16, APART), ([1000, 100, 100], 12, SINGLE), ([600, 20, 20, 20], 16, SINGLE),
    ([1500, 100, 100], 16, APART), ([2000, 100, 100], 16, NEIGHBOURS)])
def test_query_tiles_of_ragged_steps(rules, lengths, heads, order):
    """Short portions beside a long one are not counted as if they were as long."""
    assert rules.query_order(max(lengths), sum(lengths), heads, len(lengths), 128, 0) == order
    assert rules.query_order(max(lengths), sum(lengths), heads, len(lengths), 256, 0) == SINGLE
    assert rules.query_order(max(lengths), sum(lengths), heads, len(lengths), 128, 1) == (order if order == SINGLE else NEIGHBOURS)


def test_tiles_that_find_an_sm_each_do_so(rules):
    rng = random.Random(3)
    for _ in range(3000):
        lengths = [rng.randint(1, rng.choice([2, 200, 3000])) for _ in range(rng.randint(1, 8))]
        heads = rng.choice([1, 2, 4, 8, 16, 28, 40])
        tiles = [-(-n // 128) for n in lengths]
        order = rules.query_order(max(lengths), sum(lengths), heads, len(lengths), 128, 0)
        if order == SINGLE:
            assert sum(tiles) * heads <= 148
        if order == APART:
            assert sum(-(-n // 2) for n in tiles) * heads <= 148
