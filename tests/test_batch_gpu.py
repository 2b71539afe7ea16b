"""Batched engine on the B200: every graph's result equals its solo solve
(and the oracle), across several super-batches, on CUDA-graph replays."""
import numpy as np
import pytest

from conftest import undirected

pytestmark = pytest.mark.gpu


def test_batch_matches_solo_and_oracle(ecl, orc):
    b = ecl.Batch()
    b.add_mix(40, n_min=50, n_max=3000, seed=5, weight_max=1 << 16)
    hub = undirected(700, [(699, i) for i in range(699)] + [(i, i + 1) for i in range(0, 100, 2)])
    hub.eweight = np.arange(1, hub.edges + 1, dtype=np.int32) % 97 + 1
    b.add(hub)
    codes = ecl.BATCH_CC | ecl.BATCH_MIS | ecl.BATCH_GC | ecl.BATCH_MST | ecl.BATCH_SCC
    b.build(codes, max_entries=30000)  # force several super-batches
    assert b.superbatches > 2
    ms0, replay0 = b.run()
    ms1, replay1 = b.run()  # CUDA-graph replay
    assert replay1, ecl.lib.ecl_last_error()
    for i in range(b.graphs):
        g = b.graph(i)
        assert np.array_equal(b.result(i, ecl.BATCH_CC), orc.cc(g)), i
        assert np.array_equal(b.result(i, ecl.BATCH_MIS), orc.mis(g)), i
        assert np.array_equal(b.result(i, ecl.BATCH_GC), orc.gc(g)), i
        assert np.array_equal(b.result(i, ecl.BATCH_SCC), orc.scc(g)), i
        inm, tot = b.result(i, ecl.BATCH_MST)
        einm, etot = orc.mst(g)
        assert tot == etot and np.array_equal(inm, einm), i
        if i % 10 == 0:  # and the solo library call agrees
            assert np.array_equal(ecl.mis(g), b.result(i, ecl.BATCH_MIS))


def test_batch_tune_keeps_results(ecl, orc):
    b = ecl.Batch()
    b.add_mix(12, n_min=500, n_max=5000, seed=9, weight_max=1 << 16)
    b.build(ecl.BATCH_CC | ecl.BATCH_MIS | ecl.BATCH_MST)
    t = b.tune(trials=1)
    assert b.tune_points > 6
    assert t.blocks_per_sm in (64, 32, 16, 8) and t.mst_light_factor in (0.75, 1.5, 3.0, 0.4)
    assert t.row_lane_max in (8, 16, 32) and t.row_chunk in (128, 256, 512, 2048)
    b.run()
    for i in range(b.graphs):
        g = b.graph(i)
        assert np.array_equal(b.result(i, ecl.BATCH_CC), orc.cc(g))
        inm, tot = b.result(i, ecl.BATCH_MST)
        assert tot == orc.mst(g)[1]


@pytest.mark.parametrize("sizes", [
    [1, 2, 1, 2049, 1, 2048, 5000, 1, 1],  # pieces of 0, 1, 4094, 4096 and 9998 entries, cut inside and at a tile's end
    [1, 1],  # no entries at all
    [3] * 1500,  # many graphs in one tile
    [40000, 2, 3],
])
def test_batch_mst_weights_at_tile_edges(ecl, orc, sizes):
    b = ecl.Batch()
    rng = np.random.default_rng(len(sizes))
    for n in sizes:  # a path: every edge is in the forest
        u = np.arange(n - 1)
        ends = np.sort(np.concatenate([u * n + u + 1, (u + 1) * n + u]))
        w = rng.integers(0, 1 << 30, size=max(n - 1, 1))
        row, col = ends // n, ends % n
        nindex = np.searchsorted(row, np.arange(n + 1)).astype(np.int32)
        b.add(ecl.Graph(nindex, col.astype(np.int32), w[np.minimum(row, col)].astype(np.int32), symmetric=True))
    b.build(ecl.BATCH_MST)
    for _ in range(2):
        b.run()
        for i in range(0, b.graphs, max(1, b.graphs // 50)):
            inm, tot = b.result(i, ecl.BATCH_MST)
            einm, etot = orc.mst(b.graph(i))
            assert tot == etot and np.array_equal(inm, einm), i


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("count", [1, 2, 33])
def test_batch_labels_with_a_large_tree_in_every_graph(ecl, orc, count, directed):
    """CC and SCC labels are ids of the vertex's own graph, wherever its
    largest component lies and whatever is left outside it."""
    rng = np.random.default_rng(100 * count + directed)
    b = ecl.Batch()
    for k in range(count):
        kind = k % 4
        if kind == 0:  # two trees of the same size, a star of 300 and vertices without entries
            n = 1800
            edges = [(i, i + 1) for i in range(100, 700)] + [(i, i + 1) for i in range(800, 1400)]
            edges += [(1400, i) for i in range(1401, 1701)]
        elif kind == 1:
            n, edges = 1, []
        elif kind == 2:  # one tree, with the hub last
            n = 9000
            edges = [(n - 1, i) for i in range(0, n - 1, 2)] + [(i, i + 1) for i in range(0, n - 2, 2)]
        else:  # about as many edges as vertices: one large and many small components
            n = 3000
            edges = [(int(u), int(v)) for u, v in rng.integers(0, n, (n // 2 + 300, 2)) if u != v]
        g = undirected(n, edges)
        g.symmetric = not directed  # unflagged, the union takes the general paths
        b.add(g)
    b.build(ecl.BATCH_CC | ecl.BATCH_SCC)
    for _ in range(2):  # (the second a replay)
        b.run()
        for i in range(b.graphs):
            g = b.graph(i)
            assert np.array_equal(b.result(i, ecl.BATCH_CC), orc.cc(g)), i
            assert np.array_equal(b.result(i, ecl.BATCH_SCC), orc.scc(g)), i
