"""GPU plain orderings vs their CPU restatement (bit-exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def oracle_graph(P, O, g):
    off, head, ln = g.csr(True)
    return O.OGraph.from_csr(g.get_n(), off, head, ln)


@pytest.mark.parametrize("seed", [1, 99])
def test_degree_order(P, O, seed):
    g = P.Graph.rmat(12, 8, seed=4)
    og = oracle_graph(P, O, g)
    assert np.array_equal(P.Order.degree(g, seed=seed), og.degree_order(seed))


def test_degree_order_grid(P, O):
    g = P.Graph.grid(50, 40, seed=3)
    og = oracle_graph(P, O, g)
    assert np.array_equal(P.Order.degree(g, seed=7), og.degree_order(7))


@pytest.mark.parametrize("sources", [1, 16, 64])
def test_betweenness_order(P, O, sources):
    g = P.Graph.grid(30, 30, highways=10, hw_steps=8, seed=5)
    og = oracle_graph(P, O, g)
    assert np.array_equal(P.Order.betweenness(g, sources, seed=11), og.betweenness_order(sources, 11))


def test_betweenness_is_a_permutation(P):
    g = P.Graph.rmat(10, 8, seed=2)
    o = P.Order.betweenness(g, 32, seed=3)
    assert sorted(o.tolist()) == list(range(g.get_n()))


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 2047, 2048, 2049, 77824, 77825, 700001])
def test_sort_sizes(P, n):
    """Vertex counts at the edges of the radix sort's tiles and block ranges:
    degree descending, ties by the seeded key."""
    rng = np.random.default_rng(n)
    src = rng.integers(0, n, 2 * n).astype(np.uint32)
    dst = rng.integers(0, n, 2 * n).astype(np.uint32)
    g = P.Graph.from_arcs(n, src[src != dst], dst[src != dst], np.ones(int((src != dst).sum()), np.int32))
    deg = g.degrees(True).astype(np.int64) + g.degrees(False)
    with np.errstate(over="ignore"):
        z = np.uint64(5) * np.uint64(0x9E3779B97F4A7C15) + np.arange(n, dtype=np.uint64)
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    assert np.array_equal(P.Order.degree(g, seed=5), np.lexsort((z, -deg)))


@pytest.mark.parametrize("kind", ["path", "star", "rmat_weighted", "directed", "wide_grid", "scattered"])
def test_betweenness_shapes(P, O, kind, tmp_path):
    """Rounds of one vertex, hubs walked by a warp (more than 8 arcs, ends of
    32-arc groups), directed graphs, rounds longer than a block, and sources
    in components of their own."""
    rng = np.random.default_rng(3)
    if kind == "path":
        n, src, dst = 600, np.arange(599), np.arange(1, 600)
        w = rng.integers(1, 9, 599)
    elif kind == "star":
        n = 300
        src = np.concatenate([np.zeros(33), np.full(64, 1), np.full(9, 2), np.full(8, 3)]).astype(np.int64)
        dst = np.concatenate([np.arange(4, 37), np.arange(30, 94), np.arange(90, 99), np.arange(98, 106)])
        w = rng.integers(1, 3, src.size)
    elif kind in ("rmat_weighted", "directed"):
        n = 1 << 11
        g0 = P.Graph.rmat(11, 8, seed=6)
        off, head, _ = g0.csr(True)
        src, dst = np.repeat(np.arange(n), np.diff(off.astype(np.int64))), head.astype(np.int64)
        keep = src < dst if kind == "rmat_weighted" else rng.random(src.size) < 0.5
        src, dst = src[keep], dst[keep]
        w = rng.integers(1, 6, src.size)
    elif kind == "wide_grid":
        n = 20000
        i = np.arange(n).reshape(100, 200)
        src = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
        dst = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
        w = np.ones(src.size, np.int64)
    else:
        n, src, dst = 1000, np.arange(0, 300, 3), np.arange(1, 301, 3)
        w = rng.integers(1, 2, 100)
    g = P.Graph.from_arcs(n, src.astype(np.uint32), dst.astype(np.uint32), w.astype(np.int32),
                          undirected=kind != "directed")
    p = str(tmp_path / "g.gr")
    g.write(p)
    og = O.OGraph.read_dimacs(p) if kind == "directed" else oracle_graph(P, O, g)
    for sources in (1, 40):
        assert np.array_equal(P.Order.betweenness(g, sources, seed=7), og.betweenness_order(sources, 7))
