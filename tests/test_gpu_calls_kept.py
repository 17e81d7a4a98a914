"""Calls that every version has to answer the same way, whatever path serves them."""
from __future__ import annotations

import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, opts

pytestmark = pytest.mark.gpu

THREADS = max(1, min(32, os.cpu_count() or 1))


def test_graph_build_with_the_smallest_wait_limit(gpu, oracle_mod):
    """A wait limit of one poll is for idle warps; a build that peels on the
    whole grid (more vertices than one block holds) still finishes."""
    u, v = gpu.gen_gnp(40000, 12.0, 11)
    og = oracle_mod.Graph.from_pairs(u, v).sort_gpu_rounds()
    with gpu.Graph.from_coo(u, v, gpu.options(spin_limit=1)) as g:
        ro, ci, lab = g.export_csr()
        assert g.info()["degeneracy"] == og.degeneracy
    off, adj, olab = og.export()
    assert np.array_equal(ro.astype(np.uint64), off) and np.array_equal(ci, adj) and np.array_equal(lab, olab)


def test_light_vertices_of_an_early_hub(gpu, oracle_mod):
    """In the stored order a hub comes first and nearly all its neighbours come
    after each of its light neighbours; these must not walk its whole list (the
    degeneracy order, where the hub comes last, takes about a fifth of the time)."""
    D, later = 200000, 7
    i = np.arange(1, D + 1, dtype=np.uint32)
    u = np.concatenate([np.zeros(D, np.uint32)] + [i[:-s] for s in range(1, later + 1)])
    v = np.concatenate([i] + [i[s:] for s in range(1, later + 1)])
    o = oracle_mod.Graph.from_pairs(u, v).sort_degeneracy().mce(threads=THREADS)
    ms = {}
    for order in (gpu.ORDER_UNCHANGED, gpu.ORDER_DEGREE_DESC, gpu.ORDER_DEGENERACY):
        with gpu.Graph.from_coo(u, v, opts(gpu, order=order)) as g:
            runs = [g.solve(opts(gpu, blocks_per_sm=4)) for _ in range(5)]
        for r in runs:
            assert (r.count, r.checksum, r.hist, r.max_size) == (o.count, o.checksum, o.hist, o.max_size)
        ms[order] = min(r.phase_ms[3] for r in runs)
    assert max(ms.values()) < 50 * ms[gpu.ORDER_DEGENERACY], ms


def test_narrow_root_range_of_a_large_graph(gpu):
    """A few roots of 10^8 vertices cost what they cost in a small graph: a
    range visits its own vertices, not all of them."""
    ms = {}
    for pairs in (100_000, 50_000_000):
        u = np.arange(0, 2 * pairs, 2, dtype=np.uint32)
        with gpu.Graph.from_coo(u, u + 1, opts(gpu)) as g:
            assert g.info()["num_edges"] == pairs
            for begin in (0, pairs // 2, pairs - 10):
                runs = [g.solve(opts(gpu, blocks_per_sm=4, root_begin=begin, root_end=begin + 10)) for _ in range(15)]
                assert all((r.count, r.roots, r.hist) == (10, 10, {2: 10}) for r in runs)
                ms.setdefault(pairs, []).append(min(r.phase_ms[3] for r in runs))
    assert max(ms[50_000_000]) < 1.5 * max(ms[100_000]), ms


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_no_room_for_the_vertex_pass(gpu, oracle_mod, tmp_path):
    """Where the vertex pass's lists cannot be allocated, a range goes root by root."""
    u, v = gpu.gen_gnp(60000, 9.0, 17)  # more vertices than warps take singly
    o = oracle_mod.Graph.from_pairs(u, v).sort_degeneracy().mce(threads=THREADS)
    path, exe = str(tmp_path / "pairs"), str(tmp_path / "scratch_check")
    np.concatenate([u, v]).tofile(path)
    lib = os.path.join(ROOT, "rdmce_b200")
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{os.path.join(lib, 'csrc')}", f"-I{os.path.join(ROOT, 'include')}",
                    "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "cpp", "scratch_check.cc"), f"-L{lib}",
                    "-lrdmce", f"-Wl,-rpath,{lib}", "-lpthread", "-o", exe], check=True, timeout=300)
    r = subprocess.run([exe, path, str(len(u))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert f"SCRATCH OK count {o.count} checksum {o.checksum}" in r.stdout


def test_device_bytes_counts_every_array(gpu):
    """Offsets, first roots, adjacency, labels with two hashes, root pairs."""
    u, v = gpu.gen_gnp(5000, 7.0, 3)
    with gpu.Graph.from_coo(u, v, opts(gpu)) as g:
        i = g.info()
        n, m = i["num_vertices"], i["num_edges"]
        assert i["device_bytes"] == 4 * (n + 1) + 4 * (n + 1) + 8 * m + (4 + 8 + 8) * n + 8 * m


def used_at_most(gpu, u, v):
    """The most device memory a build held, stream-ordered allocations of the default pool."""
    import ctypes as C

    cu, pool, value = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_uint64(0)
    used_now, used_high = 7, 8  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, _HIGH
    gpu.Graph.from_coo(u[:10], v[:10], opts(gpu)).close()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolSetAttribute(pool, used_high, C.byref(value)) == 0  # 0 resets it
    assert cu.cuMemPoolGetAttribute(pool, used_now, C.byref(value)) == 0
    before = value.value
    gpu.Graph.from_coo(u, v, opts(gpu)).close()
    assert cu.cuMemPoolGetAttribute(pool, used_high, C.byref(value)) == 0
    return value.value - before


@pytest.mark.parametrize("shape", ["edges", "path", "gnp4", "gnp16", "rmat"])
def test_memory_of_a_graph_build(gpu, shape):
    """A build stays inside what the server sets aside for a request: 96 bytes a
    pair, 40 a vertex at most, 8 a label."""
    i = np.arange(2_000_000, dtype=np.uint32)
    u, v = {"edges": lambda: (2 * i, 2 * i + 1), "path": lambda: (i, i + 1),
            "gnp4": lambda: gpu.gen_gnp(1_000_000, 4.0, 1), "gnp16": lambda: gpu.gen_gnp(250_000, 16.0, 1),
            "rmat": lambda: gpu.gen_rmat(17, 16, 1)}[shape]()
    span = int(max(u.max(), v.max())) + 1
    assert used_at_most(gpu, u, v) < 96 * len(u) + 40 * min(span, 2 * len(u)) + 8 * span + (1 << 20)


def test_server_keeps_requests_of_many_vertices_apart(gpu):
    """Two requests of separate edges, two vertices a pair, under a budget that
    holds one of them: the second waits for the first."""
    i = np.arange(1_000_000, dtype=np.uint32)
    one = (96 + 16) * len(i) + (65 << 20)  # without the memory of the vertices
    s = gpu.Server(memory_budget=2 * one)
    try:
        ids = [s.submit(2 * i, 2 * i + 1) for _ in range(2)]
        s.drain()
        assert all(s.poll(k)[0].count == len(i) for k in ids)
        spans = sorted(s.span(k) for k in ids)
    finally:
        s.close()
    assert spans[0][1] <= spans[1][0], spans
