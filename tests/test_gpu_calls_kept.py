"""Calls that every version has to answer the same way, whatever path serves them."""
from __future__ import annotations

import os

import numpy as np
import pytest

from conftest import opts

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
