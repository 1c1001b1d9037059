"""No exchanged word of the reduced BiCGStab is replaced while another tile may still wait for it.

A tile of k_schur_resident and k_schur_stream polls a neighbour's word until its tag is exactly the one it needs, so a
word replaced too early would be waited for in vain.  What orders the accesses of different tiles is only what a tile has
to see before it goes on: its neighbours' words and the sums over all tiles.  This test writes the iteration down as
events with these edges and asks, for each word, that every reading of a value comes before the store that replaces it.

The streamed form reads the extended halos of the reduced Krylov solves, where a tile may read another's words and not the
other way round (tiles 37 and 54 of an inlet of 2.0M cells); the resident form reads Chat's, which are symmetric.
"""
import itertools
import os
import re

import pytest

import cms2d_b200

CSRC = os.path.join(os.path.dirname(cms2d_b200.__file__), "csrc")
ITERS = 6


def _stream_copies():
    src = open(os.path.join(CSRC, "cms_schur_stream.cuh")).read()
    m = re.search(r"constexpr int STR_ST_COPIES = (\d+);", src)
    if not m:
        return 1
    assert src.count("tag % STR_ST_COPIES * B.words") == 2  # the store's and the poll's copy
    return int(m.group(1))


def _program(tile):
    """One tile's events in order: ("w", word, i) a store, ("r", word, i) readings from all its neighbours, ("sum", i) its
    contribution, ("tot", i) the totals known."""
    yield "w", "st", 0, tile
    yield "r", "st", 0, tile
    yield "w", "nu", 1, tile
    yield "sum", None, 0, tile
    yield "tot", None, 0, tile
    for i in range(1, ITERS):
        yield "r", "nu", i, tile
        yield "w", "st", i, tile
        yield "sum", None, i, tile
        yield "r", "st", i, tile
        yield "tot", None, i, tile
        yield "w", "nu", i + 1, tile


def _replaced_too_early(reads, ntiles, copies):
    """Pairs (reading, store) of the same word that nothing orders; reads: {tile: tiles whose words it reads}."""
    after = {}  # event -> events that follow it at once
    for t in range(ntiles):
        ev = list(_program(t))
        for a, b in itertools.pairwise(ev):
            after.setdefault(a, set()).add(b)
        for kind, word, i, _ in ev:
            if kind == "r":
                for s in reads[t]:
                    after.setdefault(("w", word, i, s), set()).add((kind, word, i, t))
            if kind == "sum":
                for s in range(ntiles):
                    after.setdefault(("sum", None, i, t), set()).add(("tot", None, i, s))

    def reaches(a, b):
        seen, stack = {a}, [a]
        while stack:
            for e in after.get(stack.pop(), ()):
                if e == b:
                    return True
                if e not in seen:
                    seen.add(e)
                    stack.append(e)
        return False

    bad = []
    for t in range(ntiles):
        for s in reads[t]:
            for word, n in (("st", copies), ("nu", 1)):
                first = 0 if word == "st" else 1
                for i in range(first, ITERS - n):
                    if not reaches(("r", word, i, t), ("w", word, i + n, s)):
                        bad.append((word, i, t, s))
    return bad


ONE_WAY = {0: [1], 1: [], 2: []}
CHAIN = {0: [1], 1: [2], 2: []}
SYMMETRIC = {0: [1, 2], 1: [0], 2: [0]}


@pytest.mark.parametrize("reads", [ONE_WAY, CHAIN, SYMMETRIC], ids=["one_way", "chain", "symmetric"])
def test_streamed_words_are_read_before_they_are_replaced(reads):
    assert _replaced_too_early(reads, 3, _stream_copies()) == []


def test_resident_words_are_read_before_they_are_replaced():
    assert _replaced_too_early(SYMMETRIC, 3, 1) == []


def test_the_check_sees_a_missing_copy():
    assert _replaced_too_early(ONE_WAY, 3, 1) == [("st", i, 0, 1) for i in range(1, ITERS - 1)]  # (0: the sums of the start)
