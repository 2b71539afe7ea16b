"""MIS, GC, MST, SCC and APSP on the B200 vs the oracle (bit-exact)."""
import numpy as np
import pytest

from conftest import from_edges, overlapping_rows, undirected

pytestmark = pytest.mark.gpu


def sym_cases(ecl):
    yield "single", ecl.Graph(np.array([0, 0], np.int32), np.array([], np.int32), symmetric=True)
    yield "pair", undirected(2, [(0, 1)])
    yield "path", undirected(9, [(i, i + 1) for i in range(8)])
    yield "star", undirected(300, [(0, i) for i in range(1, 300)])
    yield "isolated", undirected(12, [(3, 7), (7, 9)])
    yield "clique", undirected(50, [(i, j) for i in range(50) for j in range(i + 1, 50)])
    yield "grid", ecl.gen_grid(48, 48, 0.05, seed=1)
    yield "rmat12", ecl.gen_rmat(12, 16, seed=2)
    yield "rmat14", ecl.gen_rmat(14, 8, seed=5)
    yield "er", ecl.gen_er(3000, 0.003, seed=4, symmetrise=True)
    yield "hub", undirected(9000, [(8999, i) for i in range(8999)] + [(i, i + 1) for i in range(0, 200, 2)])


def weighted(g, seed=3, wmax=1 << 20):
    """Attach pair-symmetric weights to a symmetric graph."""
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(g.nodes), np.diff(g.nindex))
    lo = np.minimum(src, g.nlist).astype(np.int64)
    hi = np.maximum(src, g.nlist).astype(np.int64)
    key = lo * (g.nodes + 1) + hi
    uniq, inv = np.unique(key, return_inverse=True)
    w = rng.integers(1, wmax, size=uniq.shape[0]).astype(np.int32)
    g.eweight = w[inv]
    return g


# ------------------------------------------------------------------------- MIS


def test_mis_matches_oracle(ecl, orc):
    for name, g in sym_cases(ecl):
        got = ecl.mis(g)
        assert np.array_equal(got, orc.mis(g)), name
        assert orc.verify_mis(g, got) == 0, name


def test_mis_device_resident(ecl, orc):
    g = ecl.gen_rmat(14, 16, seed=2)
    out = ecl.mis(g.to_device())
    assert np.array_equal(out.cpu().numpy(), orc.mis(g))


def test_mis_self_loop_is_rejected(ecl):
    """The reference spins forever on a self-loop (v never beats itself);
    here the device scan reports ECL_ERR_BAD_GRAPH, and host validation
    rejects it before any launch."""
    g = from_edges(3, [(0, 0), (0, 1), (1, 0)])
    with pytest.raises(ecl.EclError) as e:
        ecl.mis(g, max_rounds=50)
    assert e.value.status == ecl.ERR_BAD_GRAPH
    with pytest.raises(ecl.EclError) as e:
        ecl.mis(g, validate=True)
    assert e.value.status == ecl.ERR_BAD_GRAPH


# -------------------------------------------------------------------------- GC


def test_gc_matches_greedy_oracle(ecl, orc):
    for name, g in sym_cases(ecl):
        got = ecl.gc(g)
        exp = orc.gc(g)
        assert orc.verify_gc(g, got)[0] == 0, name
        assert np.array_equal(got, exp), name


def test_gc_large_colour_windows(ecl, orc):
    # a 150-clique forces colours far beyond one 64-colour window
    g = undirected(160, [(i, j) for i in range(150) for j in range(i + 1, 150)] + [(150 + k, k) for k in range(10)])
    got = ecl.gc(g)
    assert np.array_equal(got, orc.gc(g))
    assert got.max() == 149


# ------------------------------------------------------------------------- MST


@pytest.mark.parametrize("core", [1, 7, 64, 0])
@pytest.mark.parametrize("ctas", [0, 1, 4])
def test_gc_core_size_does_not_change_colours(ecl, orc, core, ctas):
    """The leading ranks are coloured in shared memory -- by a cluster of CTAs
    (two by default, one or four here) with a copy of the colours in each --
    and the rest by the grid-wide pull; where the boundary lies (1, 7, 64
    ranks, or the default of 8192) and how many CTAs colour the core change no
    colour.  A 2100-clique
    (every vertex a long row inside the default core) forces colours past the
    first 2048-colour window there."""
    old = ecl.set_tune(gc_core_ranks=core, gc_core_ctas=ctas)
    try:
        cases = list(sym_cases(ecl)) + [("rmat16", ecl.gen_rmat(16, 16, seed=3))]
        if core == 0:
            cases.append(("clique2100", undirected(2100, [(i, j) for i in range(2100) for j in range(i + 1, 2100)])))
        for name, g in cases:
            assert np.array_equal(ecl.gc(g), orc.gc(g)), (core, ctas, name)
    finally:
        ecl.set_tune(old)


def test_gc_short_row_ignores_colours_above_its_range(ecl, orc):
    """A row of <= 32 entries (one lane) whose higher neighbour is a hub with
    colour 64 or more: that colour cannot be its smallest free one and must
    not stand for a low colour (64 would alias 0 in a 64-bit mask).  A
    70-clique with one pendant vertex on every member: the members keep equal
    degrees, so their colours run 0..69, and every pendant of a member
    coloured 1..69 takes colour 0."""
    n = 70
    edges = [(i, j) for i in range(n) for j in range(i + 1, n)] + [(i, n + i) for i in range(n)]
    g = undirected(2 * n, edges)
    got = ecl.gc(g)
    exp = orc.gc(g)
    assert np.array_equal(got, exp)
    assert sorted(got[:n]) == list(range(n))
    for i in range(n):
        if got[i] >= 64:
            assert got[n + i] == 0


def test_mst_matches_kruskal(ecl, orc):
    for name, g in sym_cases(ecl):
        g = weighted(g)
        inm, tot = ecl.mst(g)
        einm, etot = orc.mst(g)
        assert tot == etot, name
        assert np.array_equal(inm, einm), name


def test_mst_ties_broken_by_edge_index(ecl, orc):
    g = ecl.gen_grid(40, 40, 0.0, seed=1)
    g.eweight = np.ones(g.edges, np.int32)  # all weights equal: (w, j) order decides
    inm, tot = ecl.mst(g)
    einm, etot = orc.mst(g)
    assert tot == etot == g.nodes - 1
    assert np.array_equal(inm, einm)


def test_mst_generated_weights_and_filter(ecl, orc):
    # avg degree >= 4 takes the light/heavy path
    g = ecl.gen_rmat(14, 16, seed=2, weight_seed=3, weight_max=1 << 20)
    for sym in (False, True):
        g.symmetric = sym
        inm, tot = ecl.mst(g)
        einm, etot = orc.mst(g)
        assert tot == etot and np.array_equal(inm, einm)


# ------------------------------------------------------------------------- SCC


def dir_cases(ecl):
    yield "cycle", from_edges(5, [(0, 1), (1, 2), (2, 0), (3, 4)])
    yield "two_cycles", from_edges(8, [(0, 1), (1, 0), (1, 2), (2, 3), (3, 4), (4, 2), (5, 6), (6, 7), (7, 5), (4, 5)])
    yield "self", from_edges(3, [(0, 0), (1, 2), (2, 1), (2, 2)])
    yield "dag", from_edges(6, [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5), (0, 5)])
    yield "rmat12d", ecl.gen_rmat(12, 16, seed=2, symmetrise=False)
    yield "rmat15d", ecl.gen_rmat(15, 8, seed=7, symmetrise=False)
    yield "er_d", ecl.gen_er(4000, 0.0008, seed=4)
    yield "sym", ecl.gen_rmat(11, 8, seed=3)


def test_scc_matches_tarjan(ecl, orc):
    for name, g in dir_cases(ecl):
        got = ecl.scc(g)
        assert np.array_equal(got, orc.scc(g)), name


def giant_cases(ecl):
    """Directed graphs against the giant-component step: found, given up, with
    long rows, and with what is left for the propagation sweeps."""
    for d in (0.5, 1.2, 2.0, 6.0):
        yield f"er{d}", ecl.gen_er(6000, d / 6000, seed=int(d * 10))
    yield "rmat13", ecl.gen_rmat(13, 8, seed=3, symmetrise=False)
    yield "self_loops", from_edges(64, [(i, i) for i in range(64)] + [(5, 6), (6, 5)])
    yield "star_out", from_edges(3000, [(0, i) for i in range(1, 3000)])  # a pivot nobody reaches
    cyc = lambda a, b: [(i, i + 1 if i + 1 < b else a) for i in range(a, b)]  # noqa: E731
    yield "cycle39", from_edges(39, cyc(0, 39))  # the last length that the level limit allows, and more
    yield "cycle40", from_edges(40, cyc(0, 40))
    yield "cycle41", from_edges(41, cyc(0, 41))
    yield "cycle5000", from_edges(5000, cyc(0, 5000))
    # the pivot's component, one upstream, one downstream, one apart
    e = cyc(0, 20) + cyc(20, 35) + cyc(35, 50) + cyc(50, 64)
    yield "bowtie", from_edges(70, sorted(e + [(0, j) for j in range(2, 20)] + [(25, 3), (7, 40), (20, 45), (66, 50), (63, 67)]))
    rng = np.random.default_rng(1)  # rows just below, at and above the chunk record length
    hubs = [(h, int(x)) for h, k in ((0, 1023), (1, 1024), (2, 1025), (3, 5000)) for x in rng.permutation(9000)[:k]]
    yield "hubs", from_edges(9000, sorted(hubs + [(int(a), int(b)) for a, b in rng.integers(0, 9000, (12000, 2))]))


def test_scc_giant_component(ecl, orc):
    for name, g in giant_cases(ecl):
        exp = orc.scc(g)
        assert np.array_equal(ecl.scc(g.to_device()).cpu().numpy(), exp), name
        # every entry many times over: the same components, and entries enough
        # (2^20) for the giant-component step
        r = (1 << 20) // g.edges + 1
        big = ecl.Graph(g.nindex * r, np.repeat(g.nlist, r), None)
        assert np.array_equal(ecl.scc(big.to_device()).cpu().numpy(), exp), name


def flat_cases():
    """Rows against the 256-entry tiles of the entry-balanced scans, and average
    degrees on both sides of the MST light-edge rule."""
    yield "ring", undirected(128, [(i, (i + 1) % 128) for i in range(128)])  # rows end exactly on a tile's end
    yield "ring129", undirected(129, [(i, (i + 1) % 129) for i in range(129)])
    yield "hub", undirected(5000, [(4999, i) for i in range(4600)] + [(0, i) for i in range(1, 700)])  # rows of many tiles
    yield "empty_run", undirected(9000, [(0, 8999), (1, 8999), (8998, 8999)])  # over 2048 empty rows in one tile
    yield "two", undirected(2, [(0, 1)])
    yield "clique48", undirected(48, [(i, j) for i in range(48) for j in range(i)])
    yield "clique600", undirected(600, [(i, j) for i in range(600) for j in range(i)])


def test_mst_at_scan_tile_edges(ecl, orc):
    import torch

    for name, g in flat_cases():
        rng = np.random.default_rng(g.edges)
        for weight_max in (2, 1000):  # ties everywhere, and few
            row = np.repeat(np.arange(g.nodes), np.diff(g.nindex))
            w = rng.integers(1, weight_max, size=(g.nodes, 1 + g.nodes % 97)).astype(np.int32)
            lo, hi = np.minimum(row, g.nlist), np.maximum(row, g.nlist)
            g.eweight = w[lo, hi % w.shape[1]].astype(np.int32)
            flags, total = orc.mst(g)
            dg = g.to_device()
            got, t = ecl.mst(dg)
            assert t == total and np.array_equal(got.cpu().numpy(), flags), (name, weight_max)
            dg.nlist = torch.cat((dg.nlist[:1], dg.nlist))[1:]  # entries off the 16-byte boundaries
            got, t = ecl.mst(dg)
            assert t == total and np.array_equal(got.cpu().numpy(), flags), (name, weight_max)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 8191])  # partial groups and warps without any
def test_mis_item_lists(ecl, orc, n):
    graphs = [ecl.gen_er(n, min(1.0, d / n), seed=n + d, symmetrise=True) for d in (1, 6, 16, 17)]
    graphs.append(undirected(n, [(i, i + 1) for i in range(n - 1)]))  # long chains of decisions
    if n > 40:  # lists of 16 and 17 entries, and a hub past one 128-entry step
        graphs.append(undirected(n, [(0, i) for i in range(1, min(n, 300))] +
                                 [(1 + i, 20 + j) for i in range(8) for j in range(15 + i % 3)]))
    for k, g in enumerate(graphs):
        assert np.array_equal(ecl.mis(g), orc.mis(g)), k


def flagged_cases(ecl):
    """Graphs flagged symmetric: truly so, and falsely (SCC then must not rely on it)."""
    yield "grid", ecl.gen_grid(70, 90, 0.3, seed=2)
    yield "rmat13", ecl.gen_rmat(13, 8, seed=4)
    yield "one_entry", ecl.Graph(np.array([0, 1, 1], np.int32), np.array([1], np.int32), None, True)
    yield "no_entries", ecl.Graph(np.zeros(6, np.int32), np.zeros(0, np.int32), None, True)
    d = ecl.gen_rmat(12, 8, seed=6, symmetrise=False)
    yield "directed", ecl.Graph(d.nindex, d.nlist, None, True)
    s = ecl.gen_rmat(11, 8, seed=5)
    drop = s.edges // 2  # one direction of one edge is missing
    row = int(np.searchsorted(s.nindex, drop, side="right")) - 1
    ni = s.nindex.copy()
    ni[row + 1:] -= 1
    yield "one_missing", ecl.Graph(ni, np.delete(s.nlist, drop), None, True)
    cyc = [(i, (i + 1) % 300) for i in range(300)]
    yield "cycle", from_edges(700, cyc + [(i, i) for i in range(0, 700, 7)], symmetric=True)
    # 256-entry tiles: rows that start and end on their edges, long runs of empty rows, a row of many tiles
    yield "long_run", from_edges(9000, [(0, 8999), (8999, 0)] + [(8999, i) for i in range(4000, 4800)] +
                                 [(i, 8999) for i in range(4000, 4800)], symmetric=True)
    yield "hub", undirected(20000, [(19999, i) for i in range(19000)])
    yield "exact", undirected(512, [(i, (i + 128) % 512) for i in range(256)] + [(i, (i + 64) % 512) for i in range(256)])


def test_scc_of_graphs_flagged_symmetric(ecl, orc):
    for name, g in flagged_cases(ecl):
        exp = orc.scc(g)
        assert np.array_equal(ecl.scc(g), exp), name
        dg = g.to_device()
        assert np.array_equal(ecl.scc(dg).cpu().numpy(), exp), name
        if g.edges:  # entries off the 16-byte boundaries
            import torch

            dg.nlist = torch.cat((dg.nlist[:1], dg.nlist))[1:]
            assert np.array_equal(ecl.scc(dg).cpu().numpy(), exp), name


def sort_cases(ecl):
    for n in (2, 33, 4096, 8191, 8193, 12289, 40000):  # one block; shares of a part of a tile
        yield f"er{n}", ecl.gen_er(n, min(1.0, 5.0 / n), seed=n, symmetrise=True)
    yield "grid1440k", ecl.gen_grid(1200, 1200, 0.05, seed=1)  # shares of more than one tile
    # largest degrees of one, two and three digits
    for leaves in (255, 256, 65535, 65536):
        yield f"star{leaves}", undirected(leaves + 1, [(leaves, i) for i in range(leaves)])


def test_gc_order_at_sort_edges(ecl, orc):
    for name, g in sort_cases(ecl):
        assert np.array_equal(ecl.gc(g), orc.gc(g)), name


# ------------------------------------------------------------------------ APSP


def apsp_cases(ecl):
    yield "tiny", from_edges(3, [(0, 1), (1, 2), (0, 2), (0, 2)], weights=[2, 3, 9, 7])
    yield "selfloop", from_edges(2, [(0, 0), (0, 1)], weights=[4, 1])
    yield "er200", ecl.gen_er(200, 0.02, seed=4, weight_seed=5)
    yield "er300", ecl.gen_er(300, 0.01, seed=9, weight_seed=6)
    yield "er512", ecl.gen_er(512, 0.004, seed=4, weight_seed=4)


def test_apsp_matches_fw(ecl, orc):
    for name, g in apsp_cases(ecl):
        got = ecl.apsp(g)
        assert np.array_equal(got, orc.apsp(g)), name


def test_apsp_leading_dimension_and_device(ecl, orc):
    import torch

    g = ecl.gen_er(256, 0.01, seed=11, weight_seed=12)
    exp = orc.apsp(g)
    out = np.full((256, 300), -7, np.int32)
    ecl.apsp(g, out=out, ld=300)
    assert np.array_equal(out[:, :256], exp) and np.all(out[:, 256:] == -7)
    d = ecl.apsp(g.to_device())  # n % 128 == 0, ld == n: computed in place
    assert np.array_equal(d.cpu().numpy(), exp)


def test_apsp_reference_padded_layout(ecl, orc):
    import ctypes as C

    g = ecl.gen_er(100, 0.03, seed=13, weight_seed=14)
    upper = 128
    out = np.zeros((upper, upper), np.int32)
    st = ecl.lib.ecl_compute_apsp(g.nodes, g.edges, g.nindex.ctypes.data_as(C.POINTER(C.c_int32)),
                                  g.nlist.ctypes.data_as(C.POINTER(C.c_int32)),
                                  g.eweight.ctypes.data_as(C.POINTER(C.c_int32)), out.ctypes.data_as(C.POINTER(C.c_int32)))
    assert st == 0
    assert np.array_equal(out[:100, :100], orc.apsp(g))
    assert np.all(out[100:, :] == ecl.APSP_INF) and np.all(out[:, 100:] == ecl.APSP_INF)


# one tile and its edges, two tiles, the last size with one CTA per SM and the
# first with two (tiles of 64: 20 blocks; tiles of 128: 26), the last size with
# tiles of 64 and the first with tiles of 128
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 130, 1280, 1281, 2687, 2688, 2689, 3328, 3329])
def test_apsp_at_tile_edges(ecl, orc, n):
    import torch

    g = ecl.gen_er(n, min(0.5, 6.0 / n), seed=n, weight_seed=n + 1)
    if g.edges == 0:
        g.eweight = np.zeros(0, np.int32)
    rows = np.unique(np.linspace(0, n - 1, 24).astype(np.int32))
    exp = orc.apsp_rows(g, rows)
    dg = g.to_device()
    if dg.eweight is None or g.edges == 0:
        dg.eweight = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ecl.apsp(dg)
    assert np.array_equal(got[torch.from_numpy(rows).long().cuda()].cpu().numpy(), exp)
    # rows that start off the 16-byte boundaries: never computed in place
    flat = torch.full((n * n + 1,), -7, dtype=torch.int32, device="cuda")
    ecl.apsp(dg, out=flat[1:], ld=n)
    assert int(flat[0]) == -7 and torch.equal(flat[1:].view(n, n), got)


# ---------------------------------------------------------- malformed input and wait limits


@pytest.mark.parametrize("code", ["cc", "mis", "gc", "mst", "scc"])
def test_overlapping_rows_are_rejected_on_the_device(ecl, orc, code):
    """Without host validation the kernels see the overlapping rows: each code
    reports ECL_ERR_BAD_GRAPH (chunk records beyond the buffer are counted,
    not written), and the next solve on the same device is correct."""
    g = overlapping_rows()
    with pytest.raises(ecl.EclError) as e:
        getattr(ecl, code)(g.to_device(), validate=False)
    assert e.value.status == ecl.ERR_BAD_GRAPH
    ok = ecl.gen_rmat(12, 8, seed=2, weight_seed=3)
    assert np.array_equal(ecl.cc(ok), orc.cc(ok))


def test_mis_wait_limit_reports_no_convergence_then_recovers(ecl, orc):
    """A 100k-vertex path needs many dependent sweeps; capped at max_rounds = 1
    the persistent launch gives up with ECL_ERR_NO_CONVERGENCE instead of
    sweeping on, and the next solve on the same stream is bit-exact."""
    import torch

    n = 100000
    g = undirected(n, [(i, i + 1) for i in range(n - 1)])
    dg = g.to_device()
    with pytest.raises(ecl.EclError) as e:
        ecl.mis(dg, max_rounds=1)
    assert e.value.status == ecl.ERR_NO_CONVERGENCE
    torch.cuda.synchronize()
    assert np.array_equal(ecl.mis(dg).cpu().numpy(), orc.mis(g))


def test_scc_round_limit_reports_no_convergence_then_recovers(ecl, orc):
    """A chain of 2-cycles c0 -> c1 -> ... needs one trimming round per cycle
    (only the last cycle's maximum reaches back); max_rounds = 1 stops after
    the first round with ECL_ERR_NO_CONVERGENCE, and the next solve on the
    same stream equals the oracle."""
    k = 64
    edges = []
    for c in range(k):
        a, b = 2 * c, 2 * c + 1
        edges += [(a, b), (b, a)]
        if c + 1 < k:
            edges.append((b, 2 * c + 2))
    g = from_edges(2 * k, sorted(edges))
    dg = g.to_device()
    with pytest.raises(ecl.EclError) as e:
        ecl.scc(dg, max_rounds=1)
    assert e.value.status == ecl.ERR_NO_CONVERGENCE
    assert np.array_equal(ecl.scc(dg).cpu().numpy(), orc.scc(g))


def test_cc_validate_checks_the_symmetric_flag(ecl):
    """CC's sampling path uses each entry in both directions, so with
    validation on, an asymmetric graph flagged symmetric is rejected on the
    host before any launch."""
    g = from_edges(4, [(0, 1), (2, 3), (3, 2)], symmetric=True)
    with pytest.raises(ecl.EclError) as e:
        ecl.cc(g, validate=True)
    assert e.value.status == ecl.ERR_BAD_GRAPH


@pytest.mark.parametrize("knobs", [dict(row_lane_max=1, row_chunk=128), dict(row_lane_max=8, row_chunk=512),
                                   dict(row_lane_max=32, row_chunk=8192, blocks_per_sm=2),
                                   dict(mst_light_factor=0.4, gc_core_ranks=5, gc_pull_blocks=4, gc_core_ctas=4),
                                   dict(gc_poll_ns=2048, row_vec=1, scc_sweep_batch=4, gc_pull_blocks=1, gc_core_ctas=2)])
def test_launch_knobs_never_change_results(ecl, orc, knobs):
    """Every code under non-default degree bins, grid sizes, MST split and GC
    core size gives the oracle's result (hub rows cross every chunk size)."""
    old = ecl.set_tune(**knobs)
    try:
        g = weighted(ecl.gen_rmat(15, 16, seed=2))
        hub = undirected(9000, [(8999, i) for i in range(8999)] + [(i, i + 1) for i in range(0, 200, 2)])
        for h in (g, hub):
            assert np.array_equal(ecl.cc(h), orc.cc(h)), knobs
            assert np.array_equal(ecl.mis(h), orc.mis(h)), knobs
            assert np.array_equal(ecl.gc(h), orc.gc(h)), knobs
        inm, tot = ecl.mst(g)
        einm, etot = orc.mst(g)
        assert tot == etot and np.array_equal(inm, einm), knobs
        d = ecl.gen_rmat(14, 16, seed=2, symmetrise=False)
        assert np.array_equal(ecl.scc(d), orc.scc(d)), knobs
    finally:
        ecl.set_tune(old)


def test_mst_on_arrays_that_are_not_16_byte_aligned(ecl, orc):
    """Device CSR arrays that start 4 bytes past an allocation: the scans see
    that 16-byte row loads would be misaligned and keep to 4-byte loads; the
    forest is the same."""
    import torch

    g = ecl.gen_rmat(14, 16, seed=2, weight_seed=3)
    nl = torch.empty(g.edges + 1, dtype=torch.int32, device="cuda")
    ew = torch.empty(g.edges + 1, dtype=torch.int32, device="cuda")
    nl[1:] = torch.from_numpy(g.nlist).cuda()
    ew[1:] = torch.from_numpy(g.eweight).cuda()
    dg = ecl.DeviceGraph(torch.from_numpy(g.nindex).cuda(), nl[1:], ew[1:], True)
    assert dg.nlist.data_ptr() % 16 == 4
    inm, tot = ecl.mst(dg)
    einm, etot = orc.mst(g)
    assert tot == etot and np.array_equal(inm.cpu().numpy(), einm)


@pytest.mark.parametrize("users", [1, 7])
def test_host_graphs_through_page_locked_pieces(ecl, users):
    """Pageable inputs and outputs around the smallest size that goes through
    page-locked memory, one piece, one block and several of them; and by more
    threads at once than there are blocks."""
    import threading

    import torch

    rng = np.random.default_rng(11)
    graphs = []
    for n in (65535, 65536, 262144, 262145, 1048576, 1048577, 1350001):  # labels of 4 bytes
        # a long path without a tenth of its links
        link = rng.random(n - 1) < 0.9
        deg = np.zeros(n, np.int64)
        deg[:-1] += link
        deg[1:] += link
        nindex = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
        u = np.flatnonzero(link)
        row, col = np.concatenate([u, u + 1]), np.concatenate([u + 1, u])
        nlist = col[np.lexsort((col, row))].astype(np.int32)
        w = rng.integers(1, 1 << 30, n).astype(np.int32)
        src = np.repeat(np.arange(n), deg)
        g = ecl.Graph(nindex, nlist, w[np.minimum(src, nlist)], True)
        start = np.concatenate([[True], ~link])
        want = np.maximum.accumulate(np.where(start, np.arange(n), 0))
        graphs.append((g, want, int(w[u].astype(np.int64).sum())))
    bad = []

    def user(k):
        s = torch.cuda.Stream()
        for i in range(len(graphs)):
            g, want, total = graphs[(i + k) % len(graphs)]
            labels = np.full(g.nodes, -1, np.int32)
            ecl.cc(g, out=labels, stream=s.cuda_stream)
            inm, tot = ecl.mst(g, stream=s.cuda_stream)[:2]
            src = np.repeat(np.arange(g.nodes), np.diff(g.nindex))
            once = np.asarray(inm).astype(bool)
            if not np.array_equal(labels, want) or tot != total or once.sum() != g.edges // 2:
                bad.append((k, i))
            a, b = np.minimum(src[once], g.nlist[once]), np.maximum(src[once], g.nlist[once])
            if len(np.unique(a)) != len(a) or not np.array_equal(b, a + 1):
                bad.append((k, i, "edges"))

    threads = [threading.Thread(target=user, args=(k,)) for k in range(users)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("edges", [1, 31, 1024, 1025, 2047, 2048, 2049, 40000])
def test_mst_lists_that_one_block_finishes(ecl, orc, edges):
    """Lists of at most 2048 entries are finished by one block: from the first
    round, from a later one, with many components and with one hub; equal
    weights are told apart by the entry."""
    rng = np.random.default_rng(edges)
    n = edges + 1
    chain = [(i, i + 1) for i in range(edges)]
    star = [(0, i) for i in range(1, n)]
    k = max(2, edges // 3)  # about three edges a vertex
    dense = sorted({(int(min(u, v)), int(max(u, v))) for u, v in rng.integers(0, k, (edges, 2)) if u != v}) or [(0, 1)]
    pairs = [(2 * i, 2 * i + 1) for i in range(edges // 2)] or [(0, 1)]  # nothing left after a round
    for size, e in ((n, chain), (n, star), (k, dense), (n + 1, pairs)):
        for top in (2, 1 << 30):
            w = rng.integers(1, top, len(e)).tolist()
            g = undirected(size, e, w)
            want, total = orc.mst(g)
            inm, tot = ecl.mst(g)
            assert tot == total and np.array_equal(inm, want)


def path_csr(ecl, n, w, cut=0):
    """A path 0 - 1 - ... of n vertices with weights w[i] on (i, i + 1), without
    every cut-th link."""
    u = np.arange(n - 1)
    u = u[u % cut != cut - 1] if cut else u
    row, col = np.concatenate([u, u + 1]), np.concatenate([u + 1, u])
    order = np.lexsort((col, row))
    row, col = row[order], col[order]
    nindex = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))])
    return ecl.Graph(nindex, col, np.asarray(w)[np.minimum(row, col)], True)


def best_ms(ecl, dg, code, max_rounds=0, **kw):
    """Device time of the fastest of five calls, in ms."""
    best = 1e9
    for _ in range(5):
        o = ecl.Opts()
        o.max_rounds = max_rounds
        getattr(ecl, code)(dg, opts=o, **kw)
        best = min(best, o.elapsed_ms)
    return best


@pytest.mark.parametrize("length", [31, 32, 33, 34, 35, 1024, 1025, 1026, 1100])  # around 32 steps, and 32 * 32
@pytest.mark.parametrize("falling", [False, True])
def test_mst_of_chains_as_deep_as_the_list(ecl, length, falling):
    """Weights that fall or rise along a path hook all of it in one round into
    one chain, towards the larger ids or the smaller."""
    n = max(4000 // length, 2) * length
    w = np.arange(n)[::-1] + 1 if falling else np.arange(n) + 1
    g = path_csr(ecl, n, w, cut=length)
    flags, total = ecl.mst(g)
    row = np.repeat(np.arange(n), np.diff(g.nindex))
    assert np.array_equal(flags.astype(bool), row < g.nlist)
    assert total == int(g.eweight[row < g.nlist].astype(np.int64).sum())


def test_mst_chain_of_half_a_million_is_climbed_by_all_threads(ecl):
    """One chain much longer than the launch has threads costs about the same
    whichever way it is numbered (climbed link by link: 160 ms and more)."""
    n = 500000
    rising, falling = (path_csr(ecl, n, w).to_device() for w in (np.arange(n) + 1, np.arange(n)[::-1] + 1))
    assert best_ms(ecl, falling, "mst") < 10 * best_ms(ecl, rising, "mst") + 1.0
    assert ecl.mst(falling)[1] == n * (n + 1) // 2 - 1


@pytest.mark.parametrize("kind", ["equal", "rising", "falling"])
def test_mst_chain_of_a_short_list_is_climbed_in_steps_that_double(ecl, orc, kind):
    """One block's list hooked into one chain costs no more than the rounds of
    random weights do (climbed link by link: twenty times as much)."""
    n = 2049
    rng = np.random.default_rng(3)
    w = dict(equal=np.full(n, 7), rising=np.arange(n) + 1, falling=np.arange(n)[::-1] + 1)[kind]
    g, plain = path_csr(ecl, n, w), path_csr(ecl, n, rng.permutation(n) + 1)
    want, total = orc.mst(g)
    flags, weight = ecl.mst(g)
    assert weight == total and np.array_equal(flags, want)
    assert best_ms(ecl, g.to_device(), "mst") < 3 * best_ms(ecl, plain.to_device(), "mst")


@pytest.mark.parametrize("lead", [1, 255, 256, 700])
@pytest.mark.parametrize("code", ["cc", "gc", "mst"])  # (MIS's priorities go by the entry count, these included)
def test_entries_outside_all_rows_are_not_looked_at(ecl, orc, code, lead):
    """A CSR whose first row does not start at 0 (not validated on the host):
    what stands before it and behind the last row is no part of the graph."""
    g = ecl.gen_rmat(11, 8, seed=2, weight_seed=3)
    junk = np.full(lead, 1 << 30, np.int32)
    h = ecl.Graph(g.nindex + lead, np.concatenate([junk, g.nlist, -junk]),
                  np.concatenate([-junk, g.eweight, -junk]), True)
    want, got = getattr(orc, code)(g), getattr(ecl, code)(h.to_device())
    if code == "mst":
        assert got[1] == want[1]
        want, got = want[0], got[0]
        assert not got[:lead].any() and not got[lead + g.edges:].any()
        got = got[lead: lead + g.edges]
    assert np.array_equal(got.cpu().numpy(), want)


def directed(ecl, n, u, v):
    """CSR of the entries (u, v), each once."""
    k = np.unique(np.asarray(u, np.int64) * n + np.asarray(v, np.int64))
    nindex = np.concatenate([[0], np.cumsum(np.bincount(k // n, minlength=n))])
    return ecl.Graph(nindex, k % n, None)


def hub_graph(ecl, hubs, k, back, n=3000000):
    """A pivot (0) with 2.5 M entries, on a cycle of 32 vertices, and `hubs`
    vertices below it with k entries each to vertices without any -- but that the
    last one's last entry is n - 1, which leads to the cycle if `back`."""
    rng = np.random.default_rng(hubs)
    ends = lambda size: 100 + rng.permutation(n - 101)[:size]  # noqa: E731
    u, v = [np.zeros(2500000), np.arange(32)], [ends(2500000), np.arange(1, 33) % 32]
    u, v = u + [np.full(hubs, 5)], v + [40 + np.arange(hubs)]
    for h in range(hubs):
        u.append(np.full(k - 1 if h == hubs - 1 else k, 40 + h))
        v.append(ends(u[-1].size))
    u, v = u + [[39 + hubs, n - 1]], v + [[n - 1, 7 if back else 1000]]
    return directed(ecl, n, np.concatenate(u), np.concatenate(v))


@pytest.mark.parametrize("k", [33, 1023, 1024, 1025, 1279, 1280, 1281, 5000])  # rows by lanes, by warps and in records
@pytest.mark.parametrize("back", [False, True])
def test_scc_hubs_behind_the_giant_component(ecl, orc, k, back):
    """What decides whether a hub belongs to the component is the last entry of
    its row."""
    g = hub_graph(ecl, 3, k, back)
    want = orc.scc(g)
    assert want[0] == (g.nodes - 1 if back else 31) and want[42] == (g.nodes - 1 if back else 42)
    assert np.array_equal(ecl.scc(g.to_device()).cpu().numpy(), want)


@pytest.mark.parametrize("reached", [False, True])
@pytest.mark.parametrize("back", [False, True])
def test_scc_rows_at_the_ends_of_chunk_records(ecl, orc, reached, back):
    """Rows of exactly one and two records of the search (256 entries) and of the
    mark pass (128), and one entry less and more, whose last entry decides: it
    closes a cycle of the row's vertex and, with `back`, leads to the pivot."""
    rng = np.random.default_rng(5)
    n, sizes = 1500000, [127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 512, 513]
    ends = lambda size: 100 + rng.permutation(n - 200)[:size]  # noqa: E731
    u, v = [np.zeros(1200000), np.arange(32)], [ends(1200000), np.arange(1, 33) % 32]
    for i, k in enumerate(sizes):
        u += [np.full(k, 40 + i), [n - 1 - i]]
        v += [np.append(ends(k - 1), n - 1 - i), [40 + i]]
        if reached:
            u, v = u + [[3]], v + [[40 + i]]
        if back:
            u, v = u + [[n - 1 - i]], v + [[9]]
    g = directed(ecl, n, np.concatenate(u), np.concatenate(v))
    assert [int(g.nindex[40 + i + 1] - g.nindex[40 + i]) for i in range(len(sizes))] == sizes
    want = orc.scc(g)
    assert want[40] == n - 1 and (want[0] == n - 1) == (reached and back)
    assert np.array_equal(ecl.scc(g.to_device()).cpu().numpy(), want)


def test_scc_hubs_that_do_not_reach_the_pivot_are_shared_by_all_warps(ecl):
    """Hubs of 0.5 M entries each cost a pass over their entries, not a warp's
    walk through a row in every round (that: 7 ms a row and round)."""
    few, many = (hub_graph(ecl, h, k, False).to_device() for h, k in ((1, 33), (4, 500000)))
    assert best_ms(ecl, many, "scc") < 2.0 + 5 * best_ms(ecl, few, "scc")


@pytest.mark.parametrize("flagged", [False, True])
def test_scc_reports_the_rounds_it_took(ecl, flagged):
    """opts.rounds of a solve that went through is at least one, whichever way
    it went."""
    for g in (ecl.gen_rmat(12, 8, seed=3), ecl.gen_grid(40, 50, 0.1, seed=1), ecl.gen_rmat(17, 16, seed=3)):
        o = ecl.Opts()
        ecl.scc(ecl.Graph(g.nindex, g.nlist, None, flagged).to_device(), opts=o)
        assert o.rounds >= 1


@pytest.mark.parametrize("scale", [16, 20])
def test_scc_of_a_directed_graph_flagged_symmetric_costs_the_check_alone(ecl, orc, scale):
    """The flag is checked before anything is made of it: a directed graph that
    carries it is solved as one that does not."""
    g = ecl.gen_rmat(scale, 16, seed=6, symmetrise=False)
    plain, flagged = (ecl.Graph(g.nindex, g.nlist, None, f).to_device() for f in (False, True))
    assert np.array_equal(ecl.scc(flagged).cpu().numpy(), orc.scc(g))
    assert best_ms(ecl, flagged, "scc") < 1.5 * best_ms(ecl, plain, "scc") + 0.04


@pytest.mark.parametrize("pairs", [3, 1000, 499, 500, 501])  # (4000 vertices: around a quarter as many entries)
def test_scc_of_flagged_graphs_with_hardly_any_entries(ecl, orc, pairs):
    n = 1 << 22 if pairs == 3 else 4000
    u = 2 * np.arange(pairs) + n // 3
    g = directed(ecl, n, np.concatenate([u, u + 1]), np.concatenate([u + 1, u]))
    plain, flagged = (ecl.Graph(g.nindex, g.nlist, None, f).to_device() for f in (False, True))
    assert np.array_equal(ecl.scc(flagged).cpu().numpy(), orc.scc(g))
    if n > 4000:
        assert best_ms(ecl, flagged, "scc") < 1.15 * best_ms(ecl, plain, "scc") + 0.01


def long_distance_cases(ecl):
    """Directed graphs of a million entries and more in which the search for a
    giant component takes long or finds nothing, and whether their time can be
    compared: the sweeps of the deep layers take 46 to 200 rounds, as it happens."""
    rng = np.random.default_rng(2)
    for layers, wide, deg in ((50, 2000, 20), (300, 5000, 2)):
        u = np.repeat(np.arange((layers - 1) * wide), deg)
        g = directed(ecl, layers * wide, u, (u // wide + 1) * wide + rng.integers(0, wide, u.size))
        yield f"layers{layers}", g, layers < 100
    g = ecl.gen_grid(1000, 1100, 0.05, seed=1)
    yield "grid", ecl.Graph(g.nindex, g.nlist, None, False), True
    n = 300000
    u, v = rng.integers(0, n, (2, 4 * n))
    yield "random", directed(ecl, n, u, v), True
    # 32 vertices that reach the pivot one after another, above a random graph that does not
    n = 600000
    u, v = 100 + rng.integers(0, n - 100, (2, 10 * n))
    u = np.concatenate([np.zeros(500000), np.arange(32), u])
    v = np.concatenate([100 + rng.permutation(n - 100)[:500000], np.arange(1, 33) % 32, v])
    yield "tail", directed(ecl, n, u, v), True


def test_scc_search_for_a_giant_component_gives_up_in_time(ecl, orc):
    """A limit on the rounds, which no graph here needs, solves without the
    search: with it, little time is lost (layers: four times as much)."""
    for name, g, timed in long_distance_cases(ecl):
        dg = g.to_device()
        assert np.array_equal(ecl.scc(dg).cpu().numpy(), orc.scc(g)), name
        assert not timed or best_ms(ecl, dg, "scc") < 1.25 * best_ms(ecl, dg, "scc", max_rounds=g.nodes + 1) + 0.03, name


# Bytes of scratch that each code has asked for at least since callers could keep
# one: (nodes, entries) -> bytes.
FORMER_SCRATCH = {
    "mis": {(1000, 16000): 1280, (1 << 20, 1 << 22): 1048832, (1 << 24, 1 << 20): 16777472},
    "gc": {(1000, 16000): 117760, (1 << 20, 1 << 22): 51709952, (1 << 24, 1 << 20): 545982464},
    "scc": {(1000, 16000): 1321984, (1 << 20, 1 << 22): 81267968, (1 << 24, 1 << 20): 219286784},
}


@pytest.mark.parametrize("code", ["gc", "scc"])
def test_scratch_stays_within_a_hundredth_of_what_it_was(ecl, code):
    for (n, m), former in FORMER_SCRATCH[code].items():
        assert ecl.workspace_bytes(dict(gc=ecl.GC, scc=ecl.SCC)[code], n, m) <= 1.01 * former + 4096, (n, m)


@pytest.mark.parametrize("n", [1, 33, 1000, 70001])
def test_mis_in_a_workspace_of_one_byte_a_vertex(ecl, orc, n):
    """Workspaces of the size that MIS cannot do without, of one byte less (which
    the call does not touch), and of both sides of its full size."""
    import torch

    graphs = [ecl.gen_er(n, min(1.0, 9.0 / n), seed=n, symmetrise=True), undirected(n, [(i, i + 1) for i in range(min(n, 900) - 1)]),
              undirected(n, [(0, i) for i in range(1, min(n, 700))])]
    small, full = 256 + ((n + 3) // 4 * 4 + 255) // 256 * 256, ecl.workspace_bytes(ecl.MIS, n, 1)
    for size in (small - 1, small, full - 1, full):
        ws = torch.full((size + 64,), 0x5a, dtype=torch.uint8, device="cuda")
        for g in graphs:
            got = ecl.mis(g.to_device(), workspace=ws[:size])
            assert np.array_equal(got.cpu().numpy(), orc.mis(g)), size
        assert bool((ws[size:] == 0x5a).all()) and bool((ws == 0x5a).all()) == (size < small)


def test_server_takes_a_mis_request_that_fits_with_one_byte_a_vertex(ecl, orc):
    g = ecl.gen_rmat(16, 8, seed=7)
    resident = 4 * (g.nodes + 1) + 4 * g.edges
    out = np.zeros(g.nodes, np.uint8)
    for room, status in ((2 * g.nodes + 512, ecl.OK), (2 * g.nodes, ecl.ERR_OOM), (30 * g.nodes, ecl.OK)):
        srv = ecl.Server(slots=2, hbm_budget_bytes=resident + room)
        gid = srv.add_graph(g)
        out[:] = 7
        rc, arr, st = srv.run([(ecl.MIS, gid, 0.0, out.ctypes.data)])
        assert arr[0].status == status
        assert status != ecl.OK or (np.array_equal(out, orc.mis(g)) and st.peak_bytes <= resident + room)


def caterpillar(ecl, spine, leaves):
    """A path of `spine` vertices with `leaves` vertices of degree one at each."""
    s = np.arange(spine)
    u = np.concatenate([s[:-1], np.repeat(s, leaves)])
    v = np.concatenate([s[1:], spine + np.arange(spine * leaves)])
    g = directed(ecl, spine * (leaves + 1), np.concatenate([u, v]), np.concatenate([v, u]))
    g.symmetric = True
    return g


@pytest.mark.parametrize("leaves", [13, 14, 15, 22, 29, 30, 31])  # lists of up to 16, 17, 32 and 33 entries
@pytest.mark.parametrize("spine", [7, 8, 39, 40, 1000])  # lanes of a warp that have one, around 8
def test_mis_lists_of_middle_length(ecl, orc, spine, leaves):
    g = caterpillar(ecl, spine, leaves)
    assert np.array_equal(ecl.mis(g), orc.mis(g))


def test_mis_lists_of_middle_length_are_scanned_side_by_side(ecl):
    """Lists of 22 entries in all lanes cost little more than lists of 16 (one
    after another by the whole warp: 1.8 times as much)."""
    short, middle = (best_ms(ecl, caterpillar(ecl, 20000, k).to_device(), "mis") for k in (14, 20))
    assert middle < 1.6 * short


def clique(ecl, n, extra=0):
    """All pairs of n vertices; vertices n .. n + extra - 1 on a path behind them."""
    u, v = np.triu_indices(n, 1)
    w = n - 1 + np.arange(extra)
    u, v = np.concatenate([u, w]), np.concatenate([v, w + 1])
    return directed(ecl, n + extra, np.concatenate([u, v]), np.concatenate([v, u]))


@pytest.mark.parametrize("n", [33, 511, 513, 1015, 1017, 2030, 2031, 2032, 2033, 2034, 2035, 2049, 4064, 4066, 5000])
def test_gc_of_cliques_around_the_windows_of_colours(ecl, orc, n):
    """A clique needs as many colours as it has vertices: rows whose colour lies
    at the ends of the core's windows (of 2032 colours) and past the second."""
    g = clique(ecl, n, extra=n % 7)
    for d in (g, ecl.Graph(g.nindex, g.nlist, None, True)):
        assert np.array_equal(ecl.gc(d), orc.gc(g))


def multipartite(ecl, n, parts):
    """All pairs of n vertices in different parts."""
    u, v = np.triu_indices(n, 1)
    q = u % parts != v % parts
    return directed(ecl, n, np.concatenate([u[q], v[q]]), np.concatenate([v[q], u[q]]))


@pytest.mark.parametrize("n,parts", [(2300, 1150), (3000, 40), (4200, 2), (4500, 700), (6200, 31)])
def test_gc_of_rows_of_more_than_two_segments(ecl, orc, n, parts):
    """Core rows of up to six segments of 1024 entries, in cores on both sides of
    the rule that keeps a list of their undecided entries."""
    g = multipartite(ecl, n, parts)
    assert np.array_equal(ecl.gc(g), orc.gc(g))
    old = ecl.set_tune(gc_core_ranks=36864)  # shorter segments
    try:
        assert np.array_equal(ecl.gc(g), orc.gc(g))
    finally:
        ecl.set_tune(old)


def test_gc_of_long_rows_is_not_scanned_on_the_chain(ecl):
    """Rows of up to four segments cost what shorter ones do for each entry (a
    segment scanned behind the last neighbour's colour: four times and more)."""
    short, long_ = (best_ms(ecl, multipartite(ecl, n, 1000).to_device(), "gc") for n in (2000, 4000))
    assert long_ < 3.3 * short


def test_gc_of_cliques_costs_a_hop_for_each_colour(ecl):
    """Twice the vertices are twice the hops, not eighteen times the time."""
    small, large = (best_ms(ecl, clique(ecl, n).to_device(), "gc") for n in (1000, 2000))
    assert large < 4 * small


@pytest.mark.parametrize("n", [1025, 65537, (1 << 20) - 1, (1 << 20) + 1025])
def test_gc_order_of_equal_degrees(ecl, orc, n):
    """One degree for all vertices: the sort's left-out digits decide between
    most neighbours, on both sides of its rule, and its runs meet block and
    tile ends."""
    ring = np.stack(((np.arange(n) - 1) % n, (np.arange(n) + 1) % n), 1)
    ring.sort(axis=1)
    g = ecl.Graph((2 * np.arange(n + 1)).astype(np.int32), ring.ravel().astype(np.int32), None, True)
    assert np.array_equal(ecl.gc(g), orc.gc(g))


def cliques(ecl, count, size, tail=0):
    """`count` cliques of `size` vertices, and `tail` vertices without entries."""
    u, v = np.triu_indices(size, 1)
    base = np.repeat(np.arange(count) * size, u.size)
    u, v = np.tile(u, count) + base, np.tile(v, count) + base
    g = directed(ecl, count * size + tail, np.concatenate([u, v]), np.concatenate([v, u]))
    g.symmetric = True
    return g


# average degrees on both sides of a lane's list (16) and of 128; groups of 4, 8, 16 and 32 vertices a warp,
# the last one whole and not
@pytest.mark.parametrize("count,size,tail", [
    (1, 18, 0), (3, 17, 1), (3, 18, 1), (4300, 18, 2), (4300, 18, 3), (8500, 18, 5), (17000, 18, 11), (1, 129, 0),
    (1, 130, 0), (3, 131, 0), (3, 131, 2), (250, 140, 5), (500, 140, 9), (900, 133, 3)])
@pytest.mark.parametrize("code", ["cc", "mis", "scc"])
def test_small_groups_of_vertices(ecl, orc, code, count, size, tail):
    g = cliques(ecl, count, size, tail)
    assert np.array_equal(getattr(ecl, code)(g), getattr(orc, code)(g))


def test_mis_of_small_dense_graphs_uses_the_whole_device(ecl):
    """With 32 vertices to a warp, 94 warps scanned the 3000 lists: five times as long."""
    u, v = np.repeat(np.arange(1500), 1500), 1500 + np.tile(np.arange(1500), 1500)
    g = directed(ecl, 3000, np.concatenate([u, v]), np.concatenate([v, u]))
    g.symmetric = True
    assert best_ms(ecl, g.to_device(), "mis") < 8 * best_ms(ecl, cliques(ecl, 40, 40).to_device(), "mis")


def test_cc_of_small_dense_graphs_uses_the_whole_device(ecl):
    """As many entries in long lists as in short ones; the long ones took twice as long."""
    few, many = (best_ms(ecl, cliques(ecl, c, k).to_device(), "cc") for c, k in ((30, 300), (2000, 40)))
    assert few < 1.5 * many
