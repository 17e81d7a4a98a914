"""Decisions on words of subsets, as the kernels make them since one-step
decisions cover up to 9 candidates, restated and checked against a direct test
of every subset.

A set of candidates is a number b (the low five) and a set of the others (a
group); the 32 sets of one group are one 32-bit word.  Each row gives the sets
it rules out as words: those it contains and, if it is itself a candidate, those
that hold it and a candidate it is not adjacent to.  What no row rules out is
R + K maximal.
"""
from __future__ import annotations

import itertools
import random

import pytest

WITH = [sum(1 << b for b in range(32) if (b >> i) & 1) for i in range(5)]


def subsets_inside(row, low):
    """Word of the sets of low candidates that the row contains."""
    sub = 1
    for k in range(low):
        if (row >> k) & 1:
            sub |= sub << (1 << k)
    return sub & 0xFFFFFFFF


def words_by_row(n, adj, xrows):
    """t0_small_sets: every row, candidate or not, gives one of two ready words."""
    low, all_sets = min(n, 5), (1 << (1 << min(n, 5))) - 1
    rows = [(adj[i], i) for i in range(n)] + [(x, None) for x in xrows]
    out = set()
    for group in range(1 << (n - low)):
        members = group << low
        dead = 0
        for row, own in rows:
            sub = subsets_inside(row, low)
            inside, outside = sub, 0
            if own is not None and own < low:
                inside |= WITH[own] & ~(sub << (1 << own))
                outside = WITH[own]
            out_row = members & ~row & ~(0 if own is None or own < low else 1 << own)
            word = outside if out_row else inside
            if own is not None and own >= low and (members >> own) & 1:
                word = 0xFFFFFFFF if out_row else ~sub
            dead |= word
        out |= {b | members for b in range(1 << low) if (all_sets & ~dead) >> b & 1}
    return out


def words_by_candidate(n, adj, xrows):
    """t0_batch and tiny_vertex: the candidates' rows in turn; what other rows
    contain is marked beforehand, group by group (tiny_vertex) or there are none."""
    low, all_sets = min(n, 5), (1 << (1 << min(n, 5))) - 1
    marked = [0] * (1 << (n - low))
    for x in xrows:
        high, group = x >> low, 0
        while True:  # the groups inside the row's high part
            marked[group] |= subsets_inside(x, low)
            group = (group - high) & high
            if not group:
                break
    out = set()
    for group in range(1 << (n - low)):
        dead = marked[group]
        for i in range(n):
            sub, high = subsets_inside(adj[i], low), adj[i] >> low
            if i < low:
                dead |= WITH[i] if group & ~high else sub | (WITH[i] & ~(sub << (1 << i)))
            else:
                own = 1 << (i - low)
                word = 0 if group & ~own & ~high else sub
                dead |= ~word if group & own else word
        out |= {b | group << low for b in range(1 << low) if (all_sets & ~dead) >> b & 1}
    return out


def directly(n, adj, xrows):
    out = set()
    for s in range(1 << n):
        members = [k for k in range(n) if (s >> k) & 1]
        if any(not (adj[i] >> j) & 1 for i, j in itertools.combinations(members, 2)):
            continue
        if any(s & ~adj[i] == 0 for i in range(n) if i not in members) or any(s & ~x == 0 for x in xrows):
            continue
        out.add(s)
    return out


@pytest.mark.parametrize("n", range(1, 10))
def test_words_of_subsets_match_every_subset_decided(n):
    rnd = random.Random(n)
    for trial in range(120):
        p = rnd.choice([0.0, 0.3, 0.6, 0.85, 1.0])
        adj = [0] * n
        for i, j in itertools.combinations(range(n), 2):
            if rnd.random() < p:
                adj[i] |= 1 << j
                adj[j] |= 1 << i
        xrows = [sum(1 << k for k in range(n) if rnd.random() < rnd.choice([0.2, 0.6, 1.0]))
                 for _ in range(rnd.choice([0, 0, 1, 4]))]
        want = directly(n, adj, xrows)
        assert words_by_row(n, adj, xrows) == want
        assert words_by_candidate(n, adj, xrows) == want
