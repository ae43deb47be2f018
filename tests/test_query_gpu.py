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


class Device:
    """Arrays in device memory through the CUDA runtime that the library uses."""

    def __init__(self):
        import ctypes as C
        self.C, self.held = C, []
        self.rt = C.CDLL("libcudart.so.13")
        self.rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
        self.rt.cudaFree.argtypes = [C.c_void_p]

    def put(self, a):
        p = self.C.c_void_p()
        assert self.rt.cudaMalloc(self.C.byref(p), self.C.c_size_t(a.nbytes)) == 0
        self.held.append(p)
        assert self.rt.cudaMemcpy(p, a.ctypes.data, a.nbytes, 1) == 0
        return p

    def get(self, p, like):
        out = np.empty_like(like)
        assert self.rt.cudaMemcpy(out.ctypes.data, p, out.nbytes, 2) == 0
        return out

    def free(self):
        for p in self.held:
            self.rt.cudaFree(p)

    def sms(self):
        v = self.C.c_int()
        assert self.rt.cudaDeviceGetAttribute(self.C.byref(v), 16, 0) == 0   # multiprocessor count
        return v.value


@pytest.mark.parametrize("more", [-1, 0, 1, 2, 3, 60001])
def test_device_query_groups(P, O, more):
    """Device pairs around the size from which a warp takes four at a time
    (64 * 32 per SM), remainders of a group included: lists of lengths at the
    edges of chunks, empty ones, vertices out of range; nothing is written past
    the last answer."""
    rng = np.random.default_rng(4)
    lens = [0, 1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 200]
    lists = []
    for i, c in enumerate(lens):
        lists.append(np.sort(rng.choice(300, c, replace=False)))
        lists.append(np.arange(c) * 7 + 1000 * (i % 2))
        lists.append(np.sort(rng.choice(4000, c, replace=False)))
    n = len(lists) // 2
    off = np.zeros(2 * n + 1, np.uint64)
    off[1:] = np.cumsum([len(h) for h in lists])
    hub = np.concatenate(lists).astype(np.uint32)
    dist = rng.integers(0, 10**6, hub.size).astype(np.int32)
    L = P.Labeling.from_csr(n, off, hub, dist)
    ref = O.OLabels.from_csr(n, off, hub, dist)
    dev = Device()
    try:
        k = dev.sms() * 64 * 32 + more
        pairs = rng.integers(0, n, (k, 2)).astype(np.uint32)
        out_of_range = rng.random(k) < 0.01
        pairs[out_of_range, rng.integers(0, 2, k)[out_of_range]] = rng.choice([n, n + 1, 2**31, 2**32 - 1])
        out = np.full(k + 64, -7, np.int32)
        dp, do = dev.put(pairs), dev.put(out)
        assert P.lib().chl_query_batch_device(L._h, dp, k, do, None) == P.CHL_OK
        got = dev.get(do, out)
    finally:
        dev.free()
    want = np.full(k, P.INFTY, np.int32)
    want[~out_of_range] = ref.query(pairs[~out_of_range])
    assert np.array_equal(got[:k], want)
    assert (got[k:] == -7).all()


@pytest.mark.parametrize("k", [65537, 196607, 196608, 196609, 400_003])
def test_query_staged_batches(P, O, k):
    """Host batches either side of the size from which they are staged whole
    (196,608 pairs), from several threads at once on the same labels."""
    import threading
    g = P.Graph.rmat(10, 8, seed=2)
    L = P.build(g, P.Order.degree(g, seed=1))
    ref = O.OLabels.from_csr(g.get_n(), *L.export())
    pairs = [P.generate_query(k, g.get_n(), seed=s) for s in range(4)]
    got = [None] * 4

    def ask(i):
        for _ in range(3):
            got[i] = P.query(L, pairs[i])

    ts = [threading.Thread(target=ask, args=(i,)) for i in range(4)]
    for x in ts:
        x.start()
    for x in ts:
        x.join()
    for p, a in zip(pairs, got):
        assert np.array_equal(a, ref.query(p))


def test_query_huge_batch_is_not_slower_per_pair(P):
    """16 M pairs cost no more each than 2 M: answers past the caches made a
    pair 1.4 times as dear while they went through the slots."""
    import time
    g = P.Graph.grid(12, 12, seed=1)
    L = P.build(g, P.Order.degree(g, seed=1))

    def per_pair(k):
        pairs = P.generate_query(k, g.get_n(), seed=1)
        best = np.inf
        for _ in range(6):
            t = time.perf_counter()
            P.query(L, pairs)
            best = min(best, time.perf_counter() - t)
        return best / k

    assert per_pair(16_000_000) < 1.2 * per_pair(2_000_000)


def test_first_queries_and_exports_at_once(P):
    """Labels from host memory are uploaded, and a build's host mirror is made,
    once and whole whichever of several threads comes first."""
    import threading
    g = P.Graph.grid(60, 60, seed=3)
    built = P.build(g, P.Order.degree(g, seed=1))
    csr = built.export()
    pairs = P.generate_query(5000, g.get_n(), seed=2)
    want, sizes = P.query(built, pairs), built.list_sizes()
    bad = []

    def run(jobs):
        gate = threading.Barrier(len(jobs))

        def work(job):
            gate.wait()
            if not job():
                bad.append(job)

        ts = [threading.Thread(target=work, args=(j,)) for j in jobs]
        for t in ts:
            t.start()
        for t in ts:
            t.join()

    for _ in range(5):
        L = P.Labeling.from_csr(g.get_n(), *csr)
        run([lambda L=L: np.array_equal(P.query(L, pairs), want)] * 12)
        B = P.build(g, P.Order.degree(g, seed=1))
        run([lambda B=B: all(np.array_equal(x, y) for x, y in zip(B.export(), csr))] * 4
            + [lambda B=B: len(B.label(7, 0)[0]) == sizes.reshape(-1, 2)[7, 0]] * 4)
    assert not bad
