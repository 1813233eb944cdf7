"""The cells' edge counts at the sizes where their histogram can go wrong: runs
and rows around a warp's 32 entries, stretches of empty rows longer than a
warp, columns around the octets that hold eight, and a column whose bins fit
no block.  Every cell must be the oracle's, density bit for bit."""
import numpy as np
import pytest

import oracle as O
from pargridcpu_b200 import MultilayerGraph, synth

pytestmark = pytest.mark.gpu


def check(layers):
    g, og = MultilayerGraph.from_pairs(layers), O.OracleGraph(layers)
    table = og.coreindex()
    # powers past FP32's and FP64's range too: the fold's maximum is then infinite
    for beta in (0.0, 1.0, 30.0, 400.0):
        ref = og.densest(table, beta)
        rec, dens = g.cells(beta)
        assert np.array_equal(rec, ref["cells"])
        assert np.array_equal(dens.view(np.uint64), ref["cell_density"].view(np.uint64))
        r = g.densest([beta])[0]
        for key in ("k", "lmd", "length", "lstar", "density"):
            assert r[key] == ref[key], (beta, key)
        assert np.float32(r["max_density_f"]) == np.float32(ref["max_density_f"])


def clique(nodes):
    i, j = np.triu_indices(len(nodes), 1)
    return np.stack([nodes[i], nodes[j]], 1).astype(np.uint32)


@pytest.mark.parametrize("L", [1, 7, 8, 9, 16, 17, 33])
def test_columns_around_octets(L):
    check(synth.chung_lu_graph(700, L, 1500, 2.3, 0.5, 80 + L).layers)


@pytest.mark.parametrize("size", [31, 32, 33, 34, 65])
def test_runs_around_a_warp(size):
    check([clique(np.arange(size)), clique(np.arange(0, 2 * size, 2)), clique(np.arange(3))])


@pytest.mark.parametrize("gap", [30, 31, 32, 33, 64, 500])
def test_rows_after_empty_rows(gap):
    # a second layer that names every node, so that the ids keep their gaps
    n = 5 * (gap + 1) + 1
    path = np.stack([np.arange(n - 1), np.arange(1, n)], 1).astype(np.uint32)
    check([clique(np.arange(0, n, gap + 1)), path])


def test_a_column_whose_bins_fit_no_block():
    rng = np.random.default_rng(9)
    some = [np.unique(rng.integers(0, 640, (40, 2)), axis=0) for _ in range(199)]
    check([clique(np.arange(640))] + [p[p[:, 0] != p[:, 1]].astype(np.uint32) for p in some])


def test_more_column_groups_than_one_launch_holds():
    # 420 columns with cores of 44 to 78: 118 groups, 64 a launch
    layers = synth.erdos_renyi_graph(120, 420, 0.55, 0.55, 77).layers
    g, og = MultilayerGraph.from_pairs(layers), O.OracleGraph(layers)
    ref = og.densest(og.coreindex(), 1.0)
    rec, dens = g.cells(1.0)
    assert np.array_equal(rec, ref["cells"])
    assert np.array_equal(dens.view(np.uint64), ref["cell_density"].view(np.uint64))
