"""Batched distance queries on the GPU vs the reference Labeling::query."""
import numpy as np
import pytest

from conftest import label_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["grid12", "grid20hw", "rmat8", "directed60", "unit_path"])
def test_query_matches_reference_answers(P, case):
    c = label_case(case)
    L = P.Labeling.read(c["labels"])
    pairs = np.loadtxt(c["pairs"], dtype=np.uint32).reshape(-1, 2)
    exp = np.loadtxt(c["dist"], dtype=np.int64)
    got = P.query(L, pairs).astype(np.int64)
    assert np.array_equal(got, exp)


def test_query_large_batch_vs_oracle(P, O):
    g = P.Graph.rmat(13, 16, seed=21)
    order = P.Order.degree(g, seed=1)
    L = P.build(g, order)
    off, hub, dist = L.export()
    ref = O.OLabels.from_csr(g.get_n(), off, hub, dist)
    pairs = P.generate_query(200_000, g.get_n(), seed=3)
    assert np.array_equal(P.query(L, pairs), ref.query(pairs))


def test_query_long_labels(P, O):
    # hand-made labels with long lists to exercise multi-chunk merges
    rng = np.random.default_rng(0)
    n = 50
    lists = []
    for x in range(2 * n):
        k = int(rng.integers(0, 300))
        hubs = np.sort(rng.choice(2000, k, replace=False)).astype(np.uint32)
        d = rng.integers(0, 10**6, k).astype(np.int32)
        lists.append((hubs, d))
    off = np.zeros(2 * n + 1, np.uint64)
    off[1:] = np.cumsum([len(h) for h, _ in lists])
    hub = np.concatenate([h for h, _ in lists])
    dist = np.concatenate([d for _, d in lists])
    L = P.Labeling.from_csr(n, off, hub, dist)
    ref = O.OLabels.from_csr(n, off, hub, dist)
    pairs = np.stack(np.meshgrid(np.arange(n), np.arange(n)), -1).reshape(-1, 2).astype(np.uint32)
    assert np.array_equal(P.query(L, pairs), ref.query(pairs))


def test_query_out_of_range_rejected(P):
    c = label_case("grid12")
    L = P.Labeling.read(c["labels"])
    with pytest.raises(P.CHLError) as e:
        P.query(L, [[0, 10**6]])
    assert e.value.status == P.CHL_ERR_INVALID


def test_empty_batch(P):
    c = label_case("grid12")
    L = P.Labeling.read(c["labels"])
    assert len(P.query(L, np.zeros((0, 2), np.uint32))) == 0


@pytest.mark.parametrize("k", [1, 2, 33, 9729, 19457, 311297, 400001])
def test_query_chunk_and_group_edges(P, O, k):
    """Lists of lengths at the edges of 32-entry chunks, equal and disjoint
    ranges among them, and pair counts at the edges of a warp's group."""
    rng = np.random.default_rng(4)
    lens = [0, 1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 200]
    lists = []
    for i, c in enumerate(lens):
        lists.append(np.sort(rng.choice(300, c, replace=False)))   # dense: many common hubs
        lists.append(np.arange(c) * 7 + 1000 * (i % 2))            # one range of two, entirely before or after
        lists.append(np.sort(rng.choice(4000, c, replace=False)))
    n = len(lists) // 2
    off = np.zeros(2 * n + 1, np.uint64)
    off[1:] = np.cumsum([len(h) for h in lists])
    hub = np.concatenate(lists).astype(np.uint32)
    dist = rng.integers(0, 10**6, hub.size).astype(np.int32)
    L = P.Labeling.from_csr(n, off, hub, dist)
    ref = O.OLabels.from_csr(n, off, hub, dist)
    pairs = rng.integers(0, n, (k, 2)).astype(np.uint32)
    assert np.array_equal(P.query(L, pairs), ref.query(pairs))


def test_query_slots_and_threads(P, O):
    """Host batches around the slot size and count (32,768 pairs, 4 slots),
    from several threads at once."""
    import threading
    g = P.Graph.rmat(10, 8, seed=2)
    L = P.build(g, P.Order.degree(g, seed=1))
    ref = O.OLabels.from_csr(g.get_n(), *L.export())
    sizes = [1, 32767, 32768, 32769, 65536, 131072, 131073, 300000]
    pairs = {k: P.generate_query(k, g.get_n(), seed=k) for k in sizes}
    want = {k: ref.query(pairs[k]) for k in sizes}
    bad = []

    def ask(seed):
        for k in np.random.default_rng(seed).permutation(sizes):
            if not np.array_equal(P.query(L, pairs[int(k)]), want[int(k)]):
                bad.append(int(k))

    ts = [threading.Thread(target=ask, args=(i,)) for i in range(12)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_export_in_pieces(P):
    """An export larger than a staging buffer (16 MB) equals the lists asked
    one by one, offsets alone included."""
    import ctypes as C
    g = P.Graph.grid(140, 140, seed=4)
    L = P.build(g, P.Order.degree(g, seed=2))
    assert L.total() // 2 * 8 > 16 << 20
    off, hub, dist = L.export()
    only = np.zeros_like(off)
    assert P.lib().chl_labels_export(L._h, only.ctypes.data_as(C.POINTER(C.c_uint64)), None, None) == 0
    assert np.array_equal(only, off)
    for v in (0, 1, 777, 10000, g.get_n() - 1):
        for side in (0, 1):
            h, d = L.label(v, side)
            s = slice(int(off[2 * v + side]), int(off[2 * v + side + 1]))
            assert np.array_equal(hub[s], h) and np.array_equal(dist[s], d)
    for a, b in zip(L.export(), (off, hub, dist)):   # from the host mirror label() made
        assert np.array_equal(a, b)


def test_export_again(P):
    """A second export (through the host mirror it makes) and later ones equal
    the first (in pieces); many pairs with one out of range are refused."""
    g = P.Graph.grid(140, 140, seed=4)
    L = P.build(g, P.Order.degree(g, seed=2))
    first = L.export()
    for _ in range(2):
        for a, b in zip(L.export(), first):
            assert np.array_equal(a, b)
    pairs = P.generate_query(700_001, g.get_n(), seed=1)
    want = P.query(L, pairs)
    assert np.array_equal(want[-1000:], P.query(L, pairs[-1000:]))
    pairs[654_321, 1] = g.get_n()
    with pytest.raises(P.CHLError):
        P.query(L, pairs)
