"""Label construction on the GPU: bit-exact against the reference's labels.

Parity targets: the golden label files printed by the reference GLL binary,
and the CPU oracle (whose GLL restatement reproduces those files byte for
byte) on larger seeded graphs.  Every build mode must give the same labels:
canonical labels are unique for a given order.
"""
import filecmp

import numpy as np
import pytest

from conftest import label_case

pytestmark = pytest.mark.gpu

MODES = {"hybrid": 0, "gll": 1, "plant": 2}
CASES = ["grid12", "grid20hw", "rmat8", "directed60", "unit_path"]


def same_labels(L, ref, n):
    a = L.export()
    b = ref.export(n)
    for x, y in zip(a, b):
        if not np.array_equal(np.asarray(x), np.asarray(y)):
            return False
    return True


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("sched", ["default", "small", "rounds", "win1", "win8"])
def test_golden_label_files(P, case, mode, sched, tmp_path):
    c = label_case(case)
    g = P.Graph.read(c["gr"])
    order = P.Order.read(c["order"])
    kw = {"small": {"first_superstep": 7, "growth": 0.3},
          # first superstep by settle rounds instead of label-correcting windows
          "rounds": {"window_target": 1},
          # windows of about 2 vertices, one warp per tree; 8 warps per tree
          "win1": {"window_target": 2, "window_warps": 1, "first_superstep": 40},
          "win8": {"window_warps": 8, "window_target": 8}}.get(sched, {})
    L = P.build(g, order, mode=MODES[mode], **kw)
    out = str(tmp_path / "gpu.labels")
    L.write(out)
    assert filecmp.cmp(out, c["labels"], shallow=False)


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("sf", [32.0, 0.05])
def test_config1_grid_matches_oracle(P, O, mode, sf):
    g = P.Graph.grid(100, 100, seed=1)
    order = P.Order.degree(g, seed=1)
    off, head, ln = g.csr(True)
    og = O.OGraph.from_csr(g.get_n(), off, head, ln)
    ref, _ = O.gll(og, order)
    L = P.build(g, order, mode=MODES[mode], sf=sf)
    assert same_labels(L, ref, g.get_n())
    st = L.stats()
    assert st["supersteps"] >= 1 and st["labels"] == ref.total()


@pytest.mark.parametrize("split", [2, 16, 300])
@pytest.mark.parametrize("kind", ["grid", "rmat"])
def test_queue_split_matches_oracle(P, O, split, kind):
    # trees whose queues are split into near and far piles give the oracle's labels
    if kind == "grid":
        g = P.Graph.grid(120, 120, highways=30, seed=6)
        order = P.Order.degree(g, seed=3)
    else:
        g = P.Graph.rmat(12, 8, seed=8)
        order = P.Order.degree(g, seed=3)
    off, head, ln = g.csr(True)
    og = O.OGraph.from_csr(g.get_n(), off, head, ln)
    ref, _ = O.gll(og, order)
    for mode in (MODES["hybrid"], MODES["gll"]):
        L = P.build(g, order, mode=mode, queue_split=split)
        assert same_labels(L, ref, g.get_n()), (split, mode)
        # the first superstep's windows sized like the split
        L = P.build(g, order, mode=mode, window_target=split, first_superstep=split * 4)
        assert same_labels(L, ref, g.get_n()), ("window", split, mode)


@pytest.mark.parametrize("mode", list(MODES))
def test_rmat_unit_lengths_matches_oracle(P, O, mode):
    g = P.Graph.rmat(12, 16, seed=5)
    order = P.Order.degree(g, seed=2)
    off, head, ln = g.csr(True)
    og = O.OGraph.from_csr(g.get_n(), off, head, ln)
    ref, _ = O.gll(og, order)
    L = P.build(g, order, mode=MODES[mode], sf=1.0)
    assert same_labels(L, ref, g.get_n())
    L = P.build(g, order, mode=MODES[mode], sf=1.0, first_superstep=1, growth=0.05)
    assert same_labels(L, ref, g.get_n())


@pytest.mark.parametrize("mode", list(MODES))
def test_directed_weighted_matches_oracle(P, O, mode, tmp_path):
    rng = np.random.default_rng(7)
    n, m = 700, 4000
    src = rng.integers(0, n, m).astype(np.uint32)
    dst = rng.integers(0, n, m).astype(np.uint32)
    keep = src != dst
    w = rng.integers(1, 50, m).astype(np.int32)
    g = P.Graph.from_arcs(n, src[keep], dst[keep], w[keep])
    assert not g.symmetric()
    p = str(tmp_path / "d.gr")
    g.write(p)
    og = O.OGraph.read_dimacs(p)
    order = og.degree_order(3)
    ref, _ = O.gll(og, order)
    L = P.build(g, order, mode=MODES[mode], sf=0.5)
    assert same_labels(L, ref, n)


def test_directed_power_law_matches_oracle(P, O, tmp_path):
    """Directed, weighted, skewed degrees (2^15 vertices, ~2^18 arcs): two
    distinct label sides at a size where supersteps, the hash probe and the
    extension all engage."""
    rng = np.random.default_rng(11)
    n, m = 1 << 15, 1 << 18
    # endpoints: half uniform, half from a Pareto tail over a permutation
    perm = rng.permutation(n).astype(np.uint32)

    def pick(k):
        z = perm[np.minimum((rng.pareto(1.2, k) * 40).astype(np.int64), n - 1)]
        u = rng.integers(0, n, k).astype(np.uint32)
        return np.where(rng.random(k) < 0.5, z, u).astype(np.uint32)

    src, dst = pick(m), pick(m)
    keep = src != dst
    w = rng.integers(1, 100, m).astype(np.int32)
    g = P.Graph.from_arcs(n, src[keep], dst[keep], w[keep])
    assert not g.symmetric()
    p = str(tmp_path / "pl.gr")
    g.write(p)
    og = O.OGraph.read_dimacs(p)
    order = og.degree_order(5)
    ref, _ = O.gll(og, order)
    for kw in ({"queue_split": 64}, {"mode": MODES["gll"], "queue_split": 16}, {"label_cap": 5000},
               {}, {"mode": MODES["gll"]}, {"first_superstep": 100, "growth": 0.5}):
        L = P.build(g, order, **kw)
        assert same_labels(L, ref, n), kw
    pairs = P.generate_query(20000, n, seed=3)
    assert np.array_equal(P.query(L, pairs), ref.query(pairs))


def test_tiny_and_disconnected(P, O):
    # isolated vertices, a 2-cycle and a single arc
    g = P.Graph.from_arcs(5, [0, 1, 3], [1, 0, 4], [2, 2, 7])
    order = np.array([4, 2, 0, 3, 1], np.uint32)
    off, head, ln = g.csr(True)
    og = O.OGraph.from_csr(5, off, head, ln)
    ref, _ = O.gll(og, order)
    for mode in MODES.values():
        L = P.build(g, order, mode=mode)
        assert same_labels(L, ref, 5)
    L = P.build(g, order)
    q = P.query(L, [[0, 1], [3, 4], [4, 3], [2, 0], [2, 2]])
    assert q.tolist() == [2, 7, P.INFTY, P.INFTY, 0]


def test_single_vertex(P):
    g = P.Graph.from_arcs(1, [], [], [])
    L = P.build(g, np.array([0], np.uint32))
    assert L.label(0, 0)[0].tolist() == [0] and L.label(0, 1)[1].tolist() == [0]


def test_bad_order_rejected(P):
    g = P.Graph.grid(5, 5, seed=1)
    n = g.get_n()
    with pytest.raises(P.CHLError) as e:
        P.build(g, np.zeros(n, np.uint32))
    assert e.value.status == P.CHL_ERR_INVALID
    with pytest.raises(P.CHLError):
        P.build(g, np.arange(n - 1, dtype=np.uint32))


def test_build_is_deterministic(P):
    g = P.Graph.grid(60, 60, highways=40, hw_steps=16, seed=9)
    order = P.Order.degree(g, seed=4)
    a = P.build(g, order, sf=0.2).export()
    for kw in ({"max_warps": 64}, {"max_warps": 8}, {"first_superstep": 1, "growth": 0.05},
               {"first_superstep": 5000, "growth": 4.0}, {"first_superstep": 3},
               {"use_graphs": 0}, {"use_graphs": 0, "mode": 1}, {"use_graphs": 1, "mode": 1},
               {"superstep_extend": 1}, {"superstep_extend": 16, "first_superstep": 9, "growth": 0.2},
               {"superstep_extend": 16, "mode": 1, "first_superstep": 9},
               {"first_superstep": 1, "growth": 0.01, "superstep_extend": 1},
               # new-label buffers far below a superstep's labels: every
               # overflowed superstep re-runs its root range
               {"label_cap": 1000}, {"label_cap": 1000, "mode": 1}, {"label_cap": 4000, "max_warps": 8},
               {"label_cap": 3000, "first_superstep": 3}, {"label_cap": 2000, "mode": 2},
               # near/far queue split at tiny queue sizes (refills, stale
               # far entries, threshold doubling and halving), and off
               {"queue_split": 1}, {"queue_split": 2}, {"queue_split": 8}, {"queue_split": 8, "mode": 1},
               {"queue_split": 33, "first_superstep": 1, "growth": 0.05}, {"queue_split": 200},
               {"queue_split": 8, "mode": 2}, {"queue_split": 8, "max_warps": 4},
               # first-superstep windows: off, tiny, large; 1, 2 and 8 warps per tree
               {"window_target": 1}, {"window_target": 2}, {"window_target": 3, "mode": 1},
               {"window_target": 100000}, {"window_warps": 1}, {"window_warps": 2, "window_target": 16},
               {"window_warps": 8, "mode": 1}, {"window_warps": 8, "first_superstep": 5000, "window_target": 5}):
        b = P.build(g, order, sf=0.2, **kw).export()
        for x, y in zip(a, b):
            assert np.array_equal(x, y), kw


def test_sampled_queries_equal_dijkstra(P, O):
    g = P.Graph.grid(80, 80, highways=30, hw_steps=20, seed=2)
    order = P.Order.degree(g, seed=6)
    L = P.build(g, order)
    off, head, ln = g.csr(True)
    og = O.OGraph.from_csr(g.get_n(), off, head, ln)
    rng = np.random.default_rng(1)
    n = g.get_n()
    for s in rng.integers(0, n, 8):
        d = og.dijkstra(int(s))
        pairs = np.stack([np.full(n, s), np.arange(n)], 1).astype(np.uint32)
        assert np.array_equal(P.query(L, pairs), d)


def test_config1_100k_queries_equal_dijkstra(P, O):
    """Config 1: 100x100 grid, degree order, 100,000 uniform (s, t) pairs
    answered by the GPU labels and by plain Dijkstra on the CPU."""
    g = P.Graph.grid(100, 100, seed=1)
    order = P.Order.degree(g, seed=1)
    L = P.build(g, order)
    n = g.get_n()
    off, head, ln = g.csr(True)
    og = O.OGraph.from_csr(n, off, head, ln)
    pairs = P.generate_query(100000, n, seed=3)
    got = P.query(L, pairs)
    exp = np.empty(len(pairs), np.int32)
    by_src = np.argsort(pairs[:, 0], kind="stable")
    srcs, first, cnt = np.unique(pairs[by_src, 0], return_index=True, return_counts=True)
    for s, a, c in zip(srcs, first, cnt):
        sel = by_src[a:a + c]
        exp[sel] = og.dijkstra(int(s))[pairs[sel, 1]]
    assert np.array_equal(got, exp)


@pytest.mark.parametrize("mode", list(MODES))
def test_root_limit_gives_the_label_prefix(P, mode):
    """A build of the roots of rank < R holds exactly the full labeling's
    entries whose hub rank is below R (labels of committed hubs are final)."""
    g = P.Graph.grid(50, 50, highways=12, hw_steps=10, seed=13)
    order = P.Order.betweenness(g, 64, seed=2)
    full_off, full_hub, full_dist = P.build(g, order, mode=MODES[mode], sf=0.5).export()
    for limit in (1, 37, 400):
        off, hub, dist = P.build(g, order, mode=MODES[mode], sf=0.5, first_superstep=16, growth=0.5,
                                 root_limit=limit).export()
        top = int(hub.max())
        assert top == limit - 1
        for i in range(off.size - 1):
            a, b = int(full_off[i]), int(full_off[i + 1])
            keep = full_hub[a:b] <= top
            assert np.array_equal(hub[off[i]:off[i + 1]], full_hub[a:b][keep])
            assert np.array_equal(dist[off[i]:off[i + 1]], full_dist[a:b][keep])


def test_unpruned_supersteps_give_way_to_pruned_ones(P, O):
    """Random sparse graphs settle far more vertices than they label: the
    whole-graph superstep ends by its settled-vertices ratio and the rest is
    pruned.  Small label budgets end it by the budget instead."""
    rng = np.random.default_rng(5)
    n = 6000
    src = np.repeat(np.arange(n), 3)
    dst = rng.integers(0, n, src.size)
    keep = src != dst
    for undirected in (True, False):
        g = P.Graph.from_arcs(n, src[keep], dst[keep], rng.integers(1, 100, int(keep.sum())), undirected=undirected)
        order = P.Order.degree(g, seed=3)
        ref = None
        for kw in ({}, {"sf": 8.0}, {"mode": MODES["plant"], "window_warps": 1}, {"window_target": 1},
                   {"window_warps": 8, "window_target": 64}, {"mode": MODES["gll"], "window_warps": 2}):
            got = P.build(g, order, **kw).export()
            ref = ref or got
            assert all(np.array_equal(x, y) for x, y in zip(got, ref)), kw
        pairs = np.stack([np.full(n, 17), np.arange(n)], 1).astype(np.uint32)
        off, head, ln = g.csr(True)
        d = np.full(n, np.inf)
        d[17] = 0
        tail = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
        for _ in range(n):
            e = d.copy()
            np.minimum.at(e, head, d[tail] + ln)
            if np.array_equal(e, d):
                break
            d = e
        L = P.build(g, order)
        assert np.array_equal(P.query(L, pairs), np.where(np.isinf(d), P.INFTY, d).astype(np.int64))


def test_distances_near_int_max(P):
    """A tentative distance past INT_MAX is no error where the final ones are
    below it; a final one is (the reference asserts it)."""
    big = 2 ** 31
    g = P.Graph.from_arcs(5, [0, 0, 0, 1, 2], [1, 2, 4, 2, 3], [1, big - 10, big - 5, 1, 100])
    order = np.array([0, 1, 2, 3, 4], np.uint32)
    for kw in ({}, {"window_target": 1}, {"mode": MODES["gll"]}, {"window_target": 100, "window_warps": 1}):
        L = P.build(g, order, **kw)
        assert P.query(L, [[0, 3], [0, 4], [1, 3]]).tolist() == [102, big - 5, 101], kw
    g = P.Graph.from_arcs(3, [0, 1, 0], [1, 2, 2], [2 ** 30, 2 ** 30, 5], undirected=True)
    for kw in ({}, {"window_target": 1}, {"mode": MODES["gll"]}):
        with pytest.raises(P.CHLError) as e:
            P.build(g, np.array([0, 1, 2], np.uint32), **kw)
        assert e.value.status == P.CHL_ERR_INVALID, kw


@pytest.mark.parametrize("kind", ["rmat", "directed", "star_path", "star_long_path"])
def test_bit_parallel_supersteps(P, O, kind, tmp_path):
    """Unit lengths and heavy tails: batches of 1,024 roots a bit each (part
    batches, several per superstep, lists above 512 arcs), then the other
    kernels; a graph deeper than 64 levels falls back to them."""
    rng = np.random.default_rng(12)
    if kind == "rmat":
        g = P.Graph.rmat(13, 12, seed=9)
        n = g.get_n()
        off, head, ln = g.csr(True)
        og = O.OGraph.from_csr(n, off, head, ln)
    else:
        if kind == "directed":
            n = 5000
            z = np.minimum((rng.pareto(0.9, 40000) * 3).astype(np.int64), n - 1)
            src, dst = z, rng.integers(0, n, 40000)
            flip = rng.random(40000) < 0.5
            src, dst = np.where(flip, src, dst), np.where(flip, dst, src)
        else:
            tail = 40 if kind == "star_path" else 150
            n = 2500
            src = np.concatenate([np.zeros(2000, np.int64), np.arange(2000, 2000 + tail)])
            dst = np.concatenate([np.arange(1, 2001), np.arange(2001, 2001 + tail)])
        keep = src != dst
        g = P.Graph.from_arcs(n, src[keep], dst[keep], np.ones(int(keep.sum()), np.int32),
                              undirected=kind != "directed")
        p = str(tmp_path / "g.gr")
        g.write(p)
        if kind == "directed":
            og = O.OGraph.read_dimacs(p)
        else:
            off, head, ln = g.csr(True)
            og = O.OGraph.from_csr(n, off, head, ln)
    order = P.Order.degree(g, seed=4)
    ref, _ = O.gll(og, order)
    for kw in ({}, {"mode": MODES["gll"]}, {"mode": MODES["plant"]}, {"first_superstep": 100}, {"first_superstep": 1025},
               {"first_superstep": 1500, "growth": 1.0}, {"sf": 0.5}, {"label_cap": 3000}, {"root_limit": n},
               {"first_superstep": 3, "growth": 0.5}, {"window_target": 1}, {"use_graphs": 0}):
        assert same_labels(P.build(g, order, **kw), ref, n), kw


@pytest.mark.parametrize("directed", [False, True])
def test_numbered_trees(P, directed):
    """Graphs of 2^16 vertices and more are renumbered for their unpruned
    trees: scrambled ids, isolated vertices and directed lengths give the
    labels of the warp-built trees."""
    side = 270
    n = side * side + 37
    rng = np.random.default_rng(8)
    i = rng.permutation(n)[:side * side].reshape(side, side)
    u = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    v = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    if directed:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
        keep = rng.random(u.size) < 0.97
        u, v = u[keep], v[keep]
    w = rng.integers(1, 1000, u.size)
    for length in (w, np.ones_like(w)):
        g = P.Graph.from_arcs(n, u, v, length, undirected=not directed)
        order = P.Order.betweenness(g, 48, seed=2)
        want = P.build(g, order, window_target=1).digest()
        assert P.build(g, order).digest() == want
        assert P.build(g, order, sf=20.0).digest() == want    # several unpruned supersteps


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n", [40, 700, 1500])
def test_rows_of_arcs(P, O, directed, n, tmp_path):
    """Weighted trees read a vertex's first four arcs as a row: degrees around
    4, 8 and 32, lists past the row, vertices without arcs, every number of
    warps per tree (32 by default on few roots)."""
    rng = np.random.default_rng(n)
    # few lists pass their row (an eighth at most): their arcs meet in a few heads
    deg = np.resize([0, 1, 2, 1], n)
    over = rng.permutation(n)[:n // 16]
    deg[over] = np.minimum(np.resize([5, 8, 9, 31, 32, 33, 36, 37, 300], over.size), n - 1)
    src = np.repeat(np.arange(n), deg)
    dst = np.where(deg[src] > 2, over[rng.integers(0, over.size, src.size)], (src + rng.integers(1, n, src.size)) % n)
    src, dst = src[src != dst], dst[src != dst]
    g = P.Graph.from_arcs(n, src, dst, rng.integers(1, 20, src.size), undirected=not directed)
    p = str(tmp_path / "g.gr")
    g.write(p)
    if directed:
        og = O.OGraph.read_dimacs(p)
    else:
        og = O.OGraph.from_csr(n, *g.csr(True))
    order = P.Order.degree(g, seed=4)
    ref, _ = O.gll(og, order)
    for kw in ({}, {"mode": MODES["gll"]}, {"mode": MODES["plant"]}, {"window_warps": 1}, {"window_warps": 2},
               {"window_warps": 4}, {"window_warps": 8, "window_target": 16}, {"first_superstep": 30}):
        assert same_labels(P.build(g, order, **kw), ref, n), kw


@pytest.mark.parametrize("mode", list(MODES))
def test_deep_unit_graphs_keep_the_trees_schedule(P, mode):
    """A heavy-tailed unit-length graph deeper than 64 levels leaves the
    bit-parallel kernel: its first superstep is then the trees' (one root per
    SM), not 2,048 roots whose trees nothing prunes."""
    g0 = P.Graph.rmat(13, 8, seed=3)
    off, head, _ = g0.csr(True)
    src, dst = np.repeat(np.arange(g0.get_n()), np.diff(off.astype(np.int64))), head.astype(np.int64)
    keep = src < dst
    n, tail = g0.get_n() + 200, np.arange(g0.get_n(), g0.get_n() + 200)
    src = np.concatenate([src[keep], [0], tail[:-1]])
    dst = np.concatenate([dst[keep], tail])
    g = P.Graph.from_arcs(n, src, dst, np.ones(src.size, np.int32), undirected=True)
    order = P.Order.degree(g, seed=1)
    L = P.build(g, order, mode=MODES[mode])
    assert L.digest() == P.build(g, order, window_target=1).digest()
    assert L.stats()["visits"] < 3_000_000
    if mode == "hybrid":
        assert L.stats()["plant_roots"] < 1024
    for kw in ({"first_superstep": 300}, {"label_cap": 2000}, {"sf": 0.5}, {"root_limit": 100}):
        a, b = P.build(g, order, mode=MODES[mode], **kw), P.build(g, order, mode=MODES[mode], window_target=1, **kw)
        assert a.digest() == b.digest(), kw


def test_bit_parallel_statistics(P):
    """Visits and arcs of bit-parallel trees, against a level-by-level search
    of every root with PLaNT's via flags; every level's launches counted."""
    rng = np.random.default_rng(3)
    n = 700
    src = np.concatenate([np.zeros(500, np.int64), rng.integers(0, n, 2500)])
    dst = np.concatenate([rng.permutation(np.arange(1, n))[:500], rng.integers(0, n, 2500)])
    keep = src != dst
    g = P.Graph.from_arcs(n, src[keep], dst[keep], np.ones(int(keep.sum()), np.int32))
    order = P.Order.degree(g, seed=2)
    rank = np.empty(n, np.int64)
    rank[order] = np.arange(n)
    st = P.build(g, order, mode=MODES["plant"]).stats()
    visits = arcs = levels = 0
    for forward in (True, False):
        off, head, _ = g.csr(forward)
        deg = np.diff(off.astype(np.int64))
        adj = np.zeros((n, n), bool)
        adj[np.repeat(np.arange(n), deg), head] = True
        depth = 0
        for r in range(n):
            seen, new, via, d = np.zeros(n, bool), np.zeros(n, bool), np.zeros(n, bool), 0
            new[order[r]] = True
            while True:
                seen |= new
                visits += int(new.sum())
                arcs += int(deg[new].sum())
                if not (new & ~via).any():
                    break
                nxt = adj[new].any(0) & ~seen
                via = nxt & (adj[new & via].any(0) | (rank < r))
                new = nxt
                d += 1
            depth = max(depth, d)
        levels += depth
    assert st["supersteps"] == 1 and (st["visits"], st["arcs"]) == (visits, arcs)
    assert st["tree_launches"] == 2 + 2 * levels


@pytest.mark.parametrize("side", [443, 444, 724, 725])
def test_window_widths_of_large_grids(P, side):
    """Either side of the sizes where windows get wider (3 * 2^16 and 2^19
    vertices): the labels of the top hubs are those of any other width."""
    g = P.Graph.grid(side, side, seed=3)
    order = P.Order.degree(g, seed=1)
    want = P.build(g, order, root_limit=300, window_target=64).digest()
    for kw in ({}, {"window_target": 512}, {"window_target": 2048, "window_warps": 4}):
        assert P.build(g, order, root_limit=300, **kw).digest() == want, kw


@pytest.mark.parametrize("directed", [False, True])
def test_numbered_trees_again_and_in_part(P, directed):
    """Renumbered graphs (2^16 vertices and more): supersteps run again after
    an overflow, ended by a root limit, and with few trees at a time."""
    side = 260
    rng = np.random.default_rng(2)
    i = rng.permutation(side * side).reshape(side, side)
    u = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    v = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    if directed:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    for length in (rng.integers(1, 100, u.size), np.ones(u.size, np.int64)):
        g = P.Graph.from_arcs(side * side, u, v, length, undirected=not directed)
        order = P.Order.betweenness(g, 48, seed=2)
        want = P.build(g, order, window_target=1, root_limit=3000).digest()
        for kw in ({}, {"label_cap": 100_000}, {"max_warps": 64}, {"sf": 3.0}, {"label_cap": 3_000_000, "max_warps": 500}):
            assert P.build(g, order, root_limit=3000, **kw).digest() == want, kw
        whole = P.build(g, order)
        assert P.build(g, order, label_cap=1_000_000).digest() == whole.digest()


def test_builds_of_several_threads(P):
    """Builds at once, whose kernels want different amounts of shared memory,
    neither fail nor change each other's labels."""
    import threading
    rng = np.random.default_rng(1)
    graphs = [P.Graph.rmat(12, 8, seed=1), P.Graph.grid(60, 60, seed=2)]
    for i, (n, m) in enumerate([(300, 1200), (2000, 20000), (4000, 16000), (900, 9000)]):
        src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
        keep = src != dst
        graphs.append(P.Graph.from_arcs(n, src[keep], dst[keep], rng.integers(1, 100, int(keep.sum())),
                                        undirected=bool(i % 2)))
    orders = [P.Order.degree(g, seed=1) for g in graphs]
    opts = [{}, {"mode": 1}, {"first_superstep": 64}, {"window_target": 1},
            {"mode": 2, "first_superstep": 50, "window_warps": 2}]
    want = [[P.build(g, o, **kw).digest() for kw in opts] for g, o in zip(graphs, orders)]
    bad = []

    def work(seed):
        r = np.random.default_rng(seed)
        for _ in range(60):
            i, j = int(r.integers(len(graphs))), int(r.integers(len(opts)))
            try:
                if P.build(graphs[i], orders[i], **opts[j]).digest() != want[i][j]:
                    bad.append((i, j, "other labels"))
            except P.CHLError as e:
                bad.append((i, j, str(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
