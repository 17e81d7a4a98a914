"""Range solves go vertex by vertex: ego networks of one root vertex at the
edges of every path (vertices decided 32 to a warp, small nodes on words of
subsets, the register tiers, the general tier, hubs left to the edge pass), and
the builder's peel at the edges of the block that finishes it, all bit-exact
against the CPU oracle."""
from __future__ import annotations

import os

import numpy as np
import pytest

from conftest import opts

pytestmark = pytest.mark.gpu

THREADS = max(1, min(32, os.cpu_count() or 1))


def assert_same(r, o):
    assert (r.count, r.checksum, r.hist, r.max_size) == (o.count, o.checksum, o.hist, o.max_size)


def ego_graph(p, x, density, seed):
    """Under the unchanged order vertex x has x earlier and p later neighbours."""
    rng = np.random.default_rng(seed)
    v0, P, X = x, np.arange(x + 1, x + 1 + p), np.arange(x)
    parts = [np.stack([np.full(p, v0), P], 1), np.stack([np.full(x, v0), X], 1)]
    i, j = np.triu_indices(p, 1)
    keep = rng.random(len(i)) < density
    parts.append(np.stack([P[i[keep]], P[j[keep]]], 1))
    a, b = np.nonzero(rng.random((x, p)) < density)
    parts.append(np.stack([X[a], P[b]], 1))
    e = np.concatenate(parts).astype(np.uint32)
    return e[:, 0].copy(), e[:, 1].copy()


@pytest.mark.parametrize("p,x,density", [
    (1, 0, 0.5), (1, 3, 0.5), (2, 1, 0.5), (5, 3, 0.5), (6, 40, 0.5), (8, 2, 0.7), (9, 60, 0.3), (10, 0, 0.6),
    (16, 16, 0.7), (31, 1, 0.6), (32, 0, 0.8), (32, 1, 0.5), (33, 5, 0.5), (40, 88, 0.4), (40, 89, 0.4),
    (50, 30, 0.05), (64, 64, 0.05), (64, 20, 0.5), (65, 10, 0.9), (200, 150, 1.0), (256, 3, 0.1), (257, 3, 0.1),
    (6, 4090, 0.5), (6, 4091, 0.5)])
def test_ego_network_of_a_root_vertex(gpu, oracle_mod, p, x, density):
    u, v = ego_graph(p, x, density, 100 * p + x)
    o = oracle_mod.Graph.from_pairs(u, v).sort_degeneracy().mce(threads=THREADS)
    with gpu.Graph.from_coo(u, v, opts(gpu, order=gpu.ORDER_UNCHANGED)) as g:
        r = g.solve(opts(gpu))
        assert r.roots == g.info()["num_edges"]
        assert_same(r, o)
        assert_same(g.solve(opts(gpu, flags=gpu.FLAG_NO_SHARING, expand_r=0)), o)


def many_components(count, seed):
    """Disjoint random graphs of 2 to 14 vertices: most vertices have few later neighbours."""
    rng = np.random.default_rng(seed)
    parts, base = [], 0
    for _ in range(count):
        n = int(rng.integers(2, 15))
        i, j = np.triu_indices(n, 1)
        keep = rng.random(len(i)) < rng.choice([0.3, 0.6, 0.95])
        parts.append(np.stack([i[keep], j[keep]], 1) + base)
        base += n
    e = np.concatenate(parts).astype(np.uint32)
    return e[:, 0].copy(), e[:, 1].copy()


@pytest.mark.parametrize("order", ["ORDER_DEGENERACY", "ORDER_UNCHANGED", "ORDER_DEGREE_DESC"])
def test_many_small_vertices(gpu, oracle_mod, order):
    """More vertices than warps take singly: the pass of 32 vertices a warp, in
    a full solve and in root ranges that cut a vertex's roots."""
    u, v = many_components(16000, 3)
    o = oracle_mod.Graph.from_pairs(u, v).sort_degeneracy().mce(threads=THREADS)
    with gpu.Graph.from_coo(u, v, opts(gpu, order=getattr(gpu, order))) as g:
        m = g.info()["num_edges"]
        r = g.solve(opts(gpu))
        assert r.roots == m
        assert_same(r, o)
        cuts = [0, m // 3 + 1, m // 2 + 1, m]
        part = [g.solve(opts(gpu, root_begin=a, root_end=b)) for a, b in zip(cuts[:-1], cuts[1:])]
    assert sum(x.count for x in part) == o.count
    assert sum(x.checksum for x in part) % (1 << 64) == o.checksum
    assert [x.roots for x in part] == [b - a for a, b in zip(cuts[:-1], cuts[1:])]


def ring_and_random(engine, n, degree, seed):
    u, v = engine.gen_gnp(n, degree, seed)
    ring = np.arange(n, dtype=np.uint32)
    return np.concatenate([u, ring]), np.concatenate([v, (ring + 1) % n]).astype(np.uint32)


@pytest.mark.parametrize("n,degree", [(2, 0.5), (4095, 1.0), (4097, 1.0), (16384, 6.0), (16385, 6.0), (6000, 510.0),
                                      (6000, 540.0), (40000, 90.0)])
def test_builder_at_its_block_edges(gpu, oracle_mod, n, degree):
    """Graphs around the sizes one block peels by itself (16384 vertices, 3 M
    neighbour entries), that reach it part-way, and around a sort tile: the
    ordered CSR equals the oracle's restatement of the peel."""
    u, v = ring_and_random(gpu, n, degree, 7) if n > 2 else (np.array([5], np.uint32), np.array([9], np.uint32))
    og = oracle_mod.Graph.from_pairs(u, v).sort_gpu_rounds()
    with gpu.Graph.from_coo(u, v, opts(gpu)) as g:
        ro, ci, lab = g.export_csr()
        assert g.info()["degeneracy"] == og.degeneracy
    off, adj, olab = og.export()
    assert np.array_equal(ro.astype(np.uint64), off)
    assert np.array_equal(ci, adj)
    assert np.array_equal(lab, olab)
