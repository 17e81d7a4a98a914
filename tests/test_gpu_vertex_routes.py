"""Which full solves go vertex by vertex first, and the vertex pass itself on
ego networks at the edges of its paths inside graphs large enough for it."""
from __future__ import annotations

import os

import numpy as np
import pytest

from conftest import opts
from test_gpu_vertex_pass import assert_same, ego_graph

pytestmark = pytest.mark.gpu

THREADS = max(1, min(32, os.cpu_count() or 1))


@pytest.mark.parametrize("p,x,density", [
    (1, 0, 0.5), (2, 1, 0.5), (5, 3, 0.5), (6, 40, 0.5), (9, 60, 0.3), (16, 16, 0.7), (31, 1, 0.6), (32, 0, 0.8),
    (32, 1, 0.5), (33, 5, 0.5), (40, 88, 0.4), (40, 89, 0.4), (50, 30, 0.05), (64, 64, 0.05), (64, 20, 0.5),
    (65, 10, 0.9), (200, 150, 1.0), (256, 3, 0.1), (257, 3, 0.1), (6, 4090, 0.5), (6, 4091, 0.5)])
def test_ego_network_among_many_vertices(gpu, oracle_mod, p, x, density):
    """The ego network of one vertex among 6000 separate edges: vertices first,
    then the roots that are left, at every build's number of warps."""
    u, v = ego_graph(p, x, density, 100 * p + x)
    i = np.arange(6000, dtype=np.uint32) * 2 + int(max(u.max(), v.max())) + 1
    u, v = np.concatenate([u, i]), np.concatenate([v, i + 1])
    o = oracle_mod.Graph.from_pairs(u, v).sort_degeneracy().mce(threads=THREADS)
    with gpu.Graph.from_coo(u, v, opts(gpu, order=gpu.ORDER_UNCHANGED)) as g:
        for blocks in (3, 4, 5):
            r = g.solve(opts(gpu, blocks_per_sm=blocks))
            assert r.launches == 2 and r.roots == g.info()["num_edges"]
            assert_same(r, o)
        for kw in (dict(expand_r=0), dict(flags=gpu.FLAG_NO_SHARING), dict(flags=gpu.FLAG_NO_SHARING, expand_r=0)):
            assert_same(g.solve(opts(gpu, **kw)), o)


@pytest.mark.parametrize("name,sharing", [("G(500, 64)", True), ("G(3000, 64)", True), ("G(6000, 150)", True),
                                          ("R-MAT 12", True), ("R-MAT 13", False), ("G(200, 100)", False),
                                          ("G(12000, 32)", False)])
def test_full_solve_is_not_slower_than_its_roots(gpu, name, sharing):
    """One warp a vertex loses to one a root where vertices are few, or dense
    without a pivot, or heavy with nobody to share them."""
    make = {"G(500, 64)": lambda: gpu.gen_gnp(500, 64.0, 1), "G(3000, 64)": lambda: gpu.gen_gnp(3000, 64.0, 1),
            "G(6000, 150)": lambda: gpu.gen_gnp(6000, 150.0, 1), "R-MAT 12": lambda: gpu.gen_rmat(12, 16, 1),
            "R-MAT 13": lambda: gpu.gen_rmat(13, 16, 1), "G(200, 100)": lambda: gpu.gen_gnp(200, 100.0, 1),
            "G(12000, 32)": lambda: gpu.gen_gnp(12000, 32.0, 1)}
    o = opts(gpu, blocks_per_sm=4, flags=0 if sharing else gpu.FLAG_NO_SHARING)
    with gpu.Graph.from_coo(*make[name](), opts(gpu)) as g:
        roots = np.arange(g.info()["num_edges"], dtype=np.uint64)
        full = [g.solve(o) for _ in range(7)]
        each = [g.solve_root_list(roots, o) for _ in range(7)]
    assert {(r.count, r.checksum) for r in full} == {(r.count, r.checksum) for r in each}
    full_ms, each_ms = (min(r.phase_ms[3] for r in rs) for rs in (full, each))
    assert full_ms < 1.4 * each_ms, (full_ms, each_ms)


def test_batch_of_dense_graphs_is_faster_than_its_roots(gpu):
    """Graphs whose mean vertex is adjacent to a third of its graph: a vertex's
    roots share most of their ego networks."""
    graphs = [gpu.gen_gnp(300, 90.0, i) for i in range(100)]
    o = opts(gpu, blocks_per_sm=4)
    b = gpu.Batch(graphs, opts(gpu))
    try:
        full = [b.solve(o) for _ in range(5)]
    finally:
        b.close()
    u, v = (np.concatenate([g[k] + 300 * i for i, g in enumerate(graphs)]).astype(np.uint32) for k in (0, 1))
    with gpu.Graph.from_coo(u, v, opts(gpu)) as g:
        roots = np.arange(g.info()["num_edges"], dtype=np.uint64)
        each = [g.solve_root_list(roots, o) for _ in range(5)]
    assert sum(r["count"] for r in full[-1][0]) == each[-1].count
    assert min(r[2] for r in full[1:]) < 0.9 * min(r.phase_ms[3] for r in each[1:])


@pytest.mark.parametrize("count,size", [(3, 200), (60, 150)])
def test_cliques_are_solved_by_vertex(gpu, oracle_mod, count, size):
    """Many later neighbours and a perfect pivot: such vertices are solved whole,
    which is far faster than each of their roots where there are vertices for
    the warps.  Cliques with some edges taken out have several maximal cliques each."""
    i, j = np.triu_indices(size, 1)
    keep = np.random.default_rng(size).random(len(i)) < 0.999
    u, v = (np.concatenate([x[keep] + size * k for k in range(count)]).astype(np.uint32) for x in (i, j))
    o = oracle_mod.Graph.from_pairs(u, v).sort_degeneracy().mce(threads=THREADS)
    with gpu.Graph.from_coo(u, v, opts(gpu)) as g:
        roots = np.arange(g.info()["num_edges"], dtype=np.uint64)
        full = [g.solve(opts(gpu, blocks_per_sm=4)) for _ in range(4)]
        each = [g.solve_root_list(roots, opts(gpu, blocks_per_sm=4)) for _ in range(4)]
        assert_same(g.solve(opts(gpu, flags=gpu.FLAG_NO_SHARING)), o)
    assert_same(full[-1], o)
    assert_same(each[-1], o)
    if count > 3:
        assert min(r.phase_ms[3] for r in full) < 0.6 * min(r.phase_ms[3] for r in each)
