"""Builds on a device with little memory (fake_device_memory.c refuses the
allocations, on the host): what is only there for speed gives way."""
import json
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, json, os, sys
import numpy as np
import plant_gb300 as P

fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_device_set.argtypes = [C.c_size_t]
fake.fake_device_live.restype = C.c_size_t
spec = json.loads(sys.argv[1])
n = spec["n"]
if spec["kind"] == "spider":
    # legs of 31 unit arcs around a centre, vertices nearer to it ranked higher:
    # every tree reaches all legs by via paths and labels little more than its own
    leg = 1 + np.arange(n - 1).reshape(-1, 31)
    src = np.concatenate([np.zeros(len(leg), np.int64), leg[:, :-1].ravel()])
    dst = np.concatenate([leg[:, 0], leg[:, 1:].ravel()])
    order = np.concatenate([[0], leg.T.ravel()]).astype(np.uint32)
    g = P.Graph.from_arcs(n, src, dst, np.ones(src.size, np.int32), undirected=True)
else:
    # disjoint pairs: next to no labels, so the graph's copies weigh most
    src = np.arange(0, n, 2)
    src, dst = np.concatenate([src, src + 1]), np.concatenate([src + 1, src])
    g = P.Graph.from_arcs(n, src, dst, 3 + (src & 1))
    order = np.random.default_rng(1).permutation(n).astype(np.uint32)
want = P.build(g, order, **spec["kw"])
got = []
if spec["kind"] == "pairs":   # host batches without room to stage them
    pairs = P.generate_query(400_000, n, seed=1)
    pairs[::3] = np.minimum(pairs[::3], n - 2) | np.array([0, 1], np.uint32)
    answers = P.query(want, pairs)
    assert (answers < P.INFTY).any()
    P.lib().chl_graph_release_device(g._h)
    fake.fake_device_set(fake.fake_device_live())
    assert np.array_equal(P.query(want, pairs), answers)
    fake.fake_device_set(C.c_size_t(-1).value)
for limit in spec["limits"]:
    fake.fake_device_set(limit + fake.fake_device_live())
    try:
        L = P.build(g, order, **spec["kw"])
        got.append([limit, "ok" if L.digest() == want.digest() else "wrong labels"])
        del L
    except P.CHLError as e:
        got.append([limit, "status %d" % e.status])
    fake.fake_device_set(C.c_size_t(-1).value)
held = fake.fake_device_live()
del want
print(json.dumps({"got": got, "held": held, "left": fake.fake_device_live()}))
"""


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    if shutil.which("gcc") is None:
        pytest.skip("no C compiler")
    so = str(tmp_path_factory.mktemp("fake") / "fake_device_memory.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", os.path.join(ROOT, "tests", "fake_device_memory.c"), "-o", so,
                    "-ldl"], check=True)
    return so


def builds(fake_lib, kind, n, limits, **kw):
    """Outcome of a build for each number of bytes the device has left."""
    spec = {"kind": kind, "n": n, "kw": kw, "limits": limits}
    r = subprocess.run([sys.executable, "-c", CHILD, json.dumps(spec)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300, env={**os.environ, "LD_PRELOAD": fake_lib})
    assert r.returncode == 0, r.stderr
    out = json.loads(r.stdout.splitlines()[-1])
    assert out["left"] == 0   # a failed build gives back what it took
    return [x for _, x in out["got"]]


def test_bit_parallel_table_that_finds_no_room(P, fake_lib):
    """The second bit-parallel superstep's table (5,500 committed roots, 32
    distances: 22.5 MB) does not fit: the trees, which need none, go on."""
    n = 1 + 500 * 31
    assert builds(fake_lib, "spider", n, [44 << 20, 52 << 20, 1 << 30], first_superstep=5500) == ["ok"] * 3
    assert builds(fake_lib, "spider", n, [16 << 20], first_superstep=5500) == ["status 3"]


@pytest.mark.parametrize("n,limits", [(1 << 17, [62 << 20, 72 << 20, 1 << 30]), (60000, [27 << 20, 31 << 20, 1 << 30])])
def test_graph_copies_that_find_no_room(P, fake_lib, n, limits):
    """The numbering (from 2^16 vertices) and the rows of arcs, or what is
    allocated after them, do not fit: the build goes on without them."""
    assert builds(fake_lib, "pairs", n, limits) == ["ok"] * 3


def test_idle_memory_is_bounded_and_given_back(P):
    """What the library keeps between calls stays below 1 GB and goes back to
    the device when a graph's device copy is released."""
    import ctypes as C
    rt = C.CDLL("libcudart.so.13")

    def free():
        f, t = C.c_size_t(), C.c_size_t()
        assert rt.cudaMemGetInfo(C.byref(f), C.byref(t)) == 0
        return f.value

    g = P.Graph.grid(300, 300, seed=1)
    order = P.Order.betweenness(g, 64, seed=1)
    P.build(g, order)
    g.release_device()
    at_first = free()
    for _ in range(3):
        P.build(g, order)
        P.Order.betweenness(g, 64, seed=1)
    assert at_first - free() <= (1 << 30) + (64 << 20)
    g.release_device()
    assert at_first - free() <= 64 << 20
