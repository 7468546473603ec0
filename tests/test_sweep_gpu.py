"""The lockstep kernel (single graphs on every SM at once) against the oracle,
at the sizes where it can go wrong: fewer rows than CTAs, rows and sources that
leave partial lanes, chunks and groups, one and two phases, degrees on both
sides of the two-level start, and grid rows in curve order."""
import numpy as np
import pytest

import odp_gb300 as og
import oracle
from conftest import same

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_small_kernel(monkeypatch):
    monkeypatch.setenv("ODP_GB300_SMALL_N", "0")


def check(spec, adjacencies):
    nd = spec.num_degrees
    b = og.Batch([spec])
    b.set_wait_limit(5 * 10 ** 9)
    for adj in adjacencies:
        want = oracle.aspl(adj, nodes=0 if spec.grid else spec.nodes, num_degrees=nd, symmetries=spec.symmetries,
                           grid=spec.grid, width=spec.width, height=spec.height)
        assert same(b.run([adj])[0], want), (spec.nodes, adj.shape, spec.symmetries, want)
    b.close()


@pytest.mark.parametrize("n,d,s", [(1, 1, 1), (2, 1, 1), (5, 3, 1), (64, 4, 4), (257, 6, 1), (600, 2, 1), (1000, 65, 1),
                                   (1217, 7, 1), (1999, 130, 1), (4104, 12, 3), (4865, 5, 1), (8192, 16, 1),
                                   (17000, 4, 1), (33333, 3, 41), (40000, 12, 1)])
def test_general_graphs(n, d, s):
    """Random directed adjacencies: d permutations of the base vertices, each
    entry turned by a random multiple of n/s."""
    rng = np.random.default_rng(n * 31 + d)
    base = n // s
    adjs = [np.stack([rng.permutation(base) + base * rng.integers(0, s, base) for _ in range(d)], axis=1).astype(np.int32)
            for _ in range(2)]
    check(og.GraphSpec(adjs[0], nodes=n, symmetries=s), adjs)


def test_ring_degrees_and_disconnection():
    n = 1500
    v = np.arange(n)
    ring = np.stack([(v + 1) % n, (v - 1) % n], axis=1).astype(np.int32)     # 750 levels
    halves = np.stack([v // 2 * 2 + (v + 1) % 2, v], axis=1).astype(np.int32)
    check(og.GraphSpec(ring, nodes=n), [ring, halves, ring])
    rng = np.random.default_rng(7)
    nd = rng.integers(1, 10, n).astype(np.int32)
    adj = rng.integers(0, n, (n, 9)).astype(np.int32)
    check(og.GraphSpec(adj, nodes=n, num_degrees=nd), [adj])


@pytest.mark.parametrize("w,h,d,length,s", [(5, 7, 4, 2, 1), (40, 40, 4, 3, 2), (36, 36, 8, 4, 4), (97, 53, 6, 4, 1),
                                            (2, 300, 4, 4, 1), (30, 30, 70, 12, 1)])
def test_grids(w, h, d, length, s):
    adjs = [og.conv_edge2adjacency_grid(w, h, og.generate_random_grid(w, h, d, length, s, seed=k), d, s)
            for k in (1, 2)]
    check(og.GraphSpec(adjs[0], grid=True, width=w, height=h, symmetries=s), adjs)


def test_grid_rows_far_apart():
    """Edges of any length: a CTA's rows have neighbours in every other CTA."""
    rng = np.random.default_rng(3)
    n = 60 * 61
    adj = rng.integers(0, n, (n, 5)).astype(np.int32)
    adj[: n // 2, 4] = np.arange(n // 2)
    check(og.GraphSpec(adj, grid=True, width=60, height=61), [adj])


def test_bad_adjacency_and_wait_limit():
    n, d = 3000, 8
    adj = og.conv_edge2adjacency_general(n, og.generate_random_general(n, d, seed=5), d)
    want = oracle.aspl(adj, nodes=n)
    b = og.Batch([og.GraphSpec(adj, nodes=n)])
    assert same(b.run()[0], want)
    bad = adj.copy()
    bad[n - 1, d - 1] = n
    with pytest.raises(og.ODPError) as e:
        b.run([bad])
    assert e.value.code == og.ERR_ADJACENCY
    b.set_wait_limit(1)                           # 1 ns: some CTA's wait for the others runs out
    with pytest.raises(og.ODPError) as e:
        b.run([adj])
    assert e.value.code == og.ERR_TIMEOUT
    b.set_wait_limit(60 * 10 ** 9)
    for _ in range(3):
        assert same(b.run([adj])[0], want)
    b.close()
