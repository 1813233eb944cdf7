"""The peel's three single-graph forms and the hand-overs between them, at the
sizes where they can go wrong: column counts around the words that hold four
columns and the segments that hold 28, rows around the 64-entry items, the
128-entry pieces and the 256-entry chunks, degrees past 16 bits, and a late
queue too short for the run.  Every table must be the oracle's, entry for
entry.

FC_PEEL_WHOLE=0 keeps a graph off the one-block and one-cluster forms;
FC_PEEL_LATE is the number of nodes at which the late form takes over (0:
never); FC_PEEL_LATE_ITEMS shortens its queues."""
import numpy as np
import pytest

import oracle as O
from pargridcpu_b200 import MultilayerGraph, batch_run, native, synth

pytestmark = pytest.mark.gpu


def check(layers, monkeypatch, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, str(v))
    ref = O.OracleGraph(layers).coreindex()
    assert np.array_equal(MultilayerGraph.from_pairs(layers).coreindex(), ref)


def graph(n, L, m, seed, gamma=2.3):
    return synth.chung_lu_graph(n, L, m, gamma, 0.4, seed).layers


@pytest.mark.parametrize("L", [1, 2, 3, 4, 5, 8, 9, 27, 28, 29, 57])
@pytest.mark.parametrize("late", [0, 700, 262144])
def test_columns_around_words_and_segments(L, late, monkeypatch):
    check(graph(1500, L, 3000, 60 + L), monkeypatch, FC_PEEL_WHOLE=0, FC_PEEL_LATE=late)


def spokes(lengths, seed):
    """Hubs with rows of exactly these lengths in one layer, over a denser
    second layer that keeps the spokes alive for some levels."""
    n = len(lengths) + max(lengths)
    star = [np.stack([np.full(k, i), len(lengths) + np.arange(k)], 1)
            for i, k in enumerate(lengths)]
    rng = np.random.default_rng(seed)
    more = rng.integers(0, n, (6 * n, 2))
    return [np.concatenate(star).astype(np.uint32), more[more[:, 0] != more[:, 1]].astype(np.uint32)]


@pytest.mark.parametrize("late", [0, 300, 262144])
def test_rows_around_items_and_chunks(late, monkeypatch):
    layers = spokes([1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 640,
                     4095, 4096, 4097], 5)
    check(layers, monkeypatch, FC_PEEL_WHOLE=0, FC_PEEL_LATE=late)


@pytest.mark.parametrize("late", [0, 40_000, 262144])
@pytest.mark.parametrize("leaves", [65_534, 65_535, 65_536, 70_001])
def test_degrees_past_sixteen_bits(leaves, late, monkeypatch):
    star = np.stack([np.zeros(leaves, np.int64), 1 + np.arange(leaves)], 1).astype(np.uint32)
    layers = [star] + graph(leaves, 2, 2 * leaves, 17)
    check(layers, monkeypatch, FC_PEEL_LATE=late)


@pytest.mark.parametrize("items", [1, 200])
def test_late_queue_too_short(items, monkeypatch):
    check(graph(4000, 6, 16_000, 23), monkeypatch, FC_PEEL_WHOLE=0, FC_PEEL_LATE_ITEMS=items)


@pytest.mark.parametrize("blocks", [4, 8, 16])
def test_cluster_sizes(blocks, monkeypatch):
    check(graph(14_000, 10, 30_000, 29), monkeypatch, FC_PEEL_CLUSTER=blocks)


@pytest.mark.parametrize("late", [0, 900, 262144])
def test_batch_with_one_layer_and_many_layer_graphs(late, monkeypatch):
    monkeypatch.setenv("FC_PEEL_LATE", str(late))
    inputs = [graph(700, 1, 2000, 31), graph(900, 30, 1500, 32), graph(1200, 4, 6000, 33),
              graph(300, 1, 500, 34)]
    tables, _, _ = batch_run([MultilayerGraph.from_pairs(x) for x in inputs])
    for layers, table in zip(inputs, tables):
        assert np.array_equal(table, O.OracleGraph(layers).coreindex())


@pytest.mark.parametrize("L", [512, 513])
def test_layers_around_what_an_entry_can_name(L, monkeypatch):
    check(graph(40, L, 60, 70 + L), monkeypatch, FC_PEEL_WHOLE=0)


@pytest.mark.parametrize("late", [None, 0])
@pytest.mark.parametrize("many", [30, 513])
@pytest.mark.parametrize("order", [1, -1])
def test_batch_of_a_one_layer_and_a_many_layer_graph(order, many, late, monkeypatch):
    """A graph that the late form cannot take does not take it from the others."""
    if late is not None:
        monkeypatch.setenv("FC_PEEL_LATE", str(late))
    inputs = [graph(700, 1, 2000, 41), graph(40, many, 60, 42), graph(900, 5, 3000, 43)][::order]
    tables, _, report = batch_run([MultilayerGraph.from_pairs(x) for x in inputs])
    assert report["peel_launches"] == (2 if many > 512 else 1)
    for layers, table in zip(inputs, tables):
        assert np.array_equal(table, O.OracleGraph(layers).coreindex())


def test_columns_that_leave_in_the_first_scan(monkeypatch):
    """Nodes with edges in few of many layers lose their higher columns at
    level 0, and with them whole words that are never written; a graph that
    used the same scratch before leaves it with other contents."""
    monkeypatch.setenv("FC_PEEL_WHOLE", "0")
    monkeypatch.setenv("FC_PEEL_LATE", "3000")
    dense = graph(4000, 12, 9000, 51)
    few = graph(4000, 3, 16_000, 52) + graph(200, 9, 900, 53)
    for layers in (dense, few, dense):
        ref = O.OracleGraph(layers).coreindex()
        assert np.array_equal(MultilayerGraph.from_pairs(layers).coreindex(), ref)


def test_deadline_is_the_whole_run_s(monkeypatch):
    """A run whose two launches each stay within the deadline and together do
    not ends with an error, and the next call gets the table."""
    gen = synth.chung_lu_graph(1_200_000, 4, 8_000_000, 2.1, 0.5, 61)
    g = MultilayerGraph.from_pairs(gen.layers)
    monkeypatch.setenv("FC_PEEL_LATE", "100000")
    ref = g.coreindex()
    times = []
    for _ in range(4):
        g.reset_results()
        g.coreindex()
        times.append(g.stats()["peel_ms"])
    limit = int(0.75 * min(times))
    assert limit >= 3
    monkeypatch.setenv("FC_PEEL_DEADLINE_MS", str(limit))
    g.reset_results()
    with pytest.raises(native.FcError) as e:
        g.coreindex()
    assert e.value.code == 6  # FC_ERR_ITER_LIMIT
    monkeypatch.delenv("FC_PEEL_DEADLINE_MS")
    assert np.array_equal(g.coreindex(), ref)


@pytest.mark.parametrize("late", [0, 2000, 262144])
def test_statistics_cover_every_form(late, monkeypatch):
    """Items and phase times of all the launches of a run, whichever form takes
    its levels."""
    monkeypatch.setenv("FC_PEEL_WHOLE", "0")
    monkeypatch.setenv("FC_PEEL_LATE", str(late))
    g = MultilayerGraph.from_pairs(graph(20_000, 5, 60_000, 62))
    ref = O.OracleGraph(graph(20_000, 5, 60_000, 62)).coreindex()
    assert np.array_equal(g.coreindex(), ref)
    st = g.stats()
    # a node is queued at least once for each level that removes it in some
    # column, unless no survivor is left that its row could name
    values = np.sort(ref, axis=0)
    removals = int((np.diff(values, axis=0) != 0).sum()) + g.n
    assert st["subrounds"] >= removals - int((ref == ref.max()).any(axis=0).sum())
    assert st["levels"] >= int(ref.max()) + 1
    scan, expand, _ = st["phase_ms"]
    assert scan > 0 and expand > 0
    assert scan + expand <= st["peel_ms"] + 0.1


@pytest.mark.parametrize("late", [None, 0, 40_000])
def test_batch_with_a_graph_of_degrees_past_sixteen_bits(late, monkeypatch):
    if late is not None:
        monkeypatch.setenv("FC_PEEL_LATE", str(late))
    leaves = 70_001
    star = np.stack([np.zeros(leaves, np.int64), 1 + np.arange(leaves)], 1).astype(np.uint32)
    inputs = [graph(900, 6, 3000, 55), [star] + graph(leaves, 2, 2 * leaves, 56),
              graph(1500, 1, 5000, 57)]
    tables, _, _ = batch_run([MultilayerGraph.from_pairs(x) for x in inputs])
    for layers, table in zip(inputs, tables):
        assert np.array_equal(table, O.OracleGraph(layers).coreindex())
