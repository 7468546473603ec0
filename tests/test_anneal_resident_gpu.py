"""The resident annealing kernel makes the moves of the stepwise kernels:
every record and graph equal after runs of several lengths, for team sizes
from one CTA up, both starts, symmetries, degree tables and grids."""
import numpy as np
import pytest

import odp_gb300 as og

pytestmark = pytest.mark.gpu


def general(n, d, s, seed):
    return og.conv_edge2adjacency_general(n, og.generate_random_general(n, d, s, seed=seed), d, s)


def grid(w, h, d, length, s, seed):
    return og.conv_edge2adjacency_grid(w, h, og.generate_random_grid(w, h, d, length, s, seed=seed), d, s)


def irregular(n, d, seed):
    adj = general(n, d, 1, seed)
    keep = np.random.default_rng(seed).random((n, n)) < 0.9
    keep &= keep.T
    nd = np.zeros(n, dtype=np.int32)
    out = np.full((n, d), -1, dtype=np.int32)
    for v in range(n):
        row = [u for u in adj[v] if keep[v, u]]
        nd[v] = len(row)
        out[v, :len(row)] = row
    return out, nd


def chains(name):
    kw = dict(max_temp=50.0, min_temp=0.5, ncalcs=200)
    if name == "small":
        return [og.Chain(general(n, d, 1, n + d), nodes=n, seed=n, **kw) for n, d in ((8, 3), (33, 4), (256, 5), (257, 12))]
    if name == "many":
        return [og.Chain(general(96, 4, 1, k), nodes=96, seed=k, **kw) for k in range(700)]
    if name == "wide":
        return [og.Chain(general(4096, 16, 1, 7), nodes=4096, seed=3, **kw),
                og.Chain(general(2000, 13, 1, 8), nodes=2000, seed=4, hill_climbing=True)]
    if name == "symmetric":
        return [og.Chain(general(n, d, s, 5), nodes=n, symmetries=s, seed=9, **kw)
                for n, d, s in ((640, 6, 2), (600, 5, 4), (1100, 8, 11))]
    adj, nd = irregular(300, 8, 6)
    return [og.Chain(adj, nodes=300, num_degrees=nd, seed=2, **kw),
            og.Chain(grid(16, 16, 4, 3, 1, 1), grid=True, width=16, height=16, length=3, seed=5, **kw),
            og.Chain(grid(12, 10, 4, 4, 2, 1), grid=True, width=12, height=10, length=4, symmetries=2, seed=6, **kw),
            og.Chain(grid(12, 12, 4, 4, 4, 1), grid=True, width=12, height=12, length=4, symmetries=4, seed=7, **kw)]


@pytest.mark.parametrize("name", ["small", "many", "wide", "symmetric", "mixed"])
def test_resident_steps_equal_the_stepwise_kernels(name, monkeypatch):
    monkeypatch.setenv("ODP_GB300_ANNEAL_RESIDENT", "1")
    a = og.Anneal(chains(name))
    monkeypatch.setenv("ODP_GB300_ANNEAL_RESIDENT", "0")
    b = og.Anneal(chains(name))
    for steps in (1, 9, 14):
        a.run(steps)
        b.run(steps)
        for k in range(len(chains("small")) if name == "many" else len(a._chains)):
            x, y = a.state(k, graphs=True), b.state(k, graphs=True)
            assert np.array_equal(x.pop("adjacency"), y.pop("adjacency")), (name, k, steps)
            assert np.array_equal(x.pop("best_adjacency"), y.pop("best_adjacency")), (name, k, steps)
            assert x == y, (name, k, steps)
    a.close()
    b.close()


@pytest.mark.parametrize("n,d,count", [(4096, 16, 1), (1500, 12, 3)])
def test_a_wait_that_runs_out_stops_the_chain(n, d, count):
    """A limit of 1 ns ends the waits of a chain's CTAs for one another: the
    chain stops with its status set, counts no step, and the state that is
    reported is the graph it holds (each edge in both its rows, at most one
    proposal away from the last one), not what its CTAs copied without having
    met."""
    kw = dict(max_temp=50.0, min_temp=0.5, ncalcs=200)
    a = og.Anneal([og.Chain(general(n, d, 1, k), nodes=n, seed=k + 1, **kw) for k in range(count)])
    a.run(6)
    before = [a.state(k, graphs=True) for k in range(count)]
    assert all(x["status"] == 0 and x["steps"] == 6 for x in before)
    a.set_wait_limit(1)
    for _ in range(2):
        a.run(3)
        for k in range(count):
            x = a.state(k, graphs=True)
            assert x["status"] == 2 and x["steps"] == 6, x["status"]
            assert np.count_nonzero(x["adjacency"] != before[k]["adjacency"]) <= 4
            assert np.array_equal(x["best_adjacency"], before[k]["best_adjacency"])
            u = np.repeat(np.arange(n), d)
            pairs = np.stack([u, x["adjacency"].ravel()])
            assert np.array_equal(np.sort(pairs[0] * n + pairs[1]), np.sort(pairs[1] * n + pairs[0]))
    a.close()


@pytest.mark.parametrize("n,d,count", [(64, 4, 3), (1024, 8, 16), (4096, 16, 1), (90, 5, 700)])
def test_a_graph_without_return_edges_stops_at_its_first_proposal(n, d, count):
    """Every thread of a team takes the same way when the proposal fails: one
    CTA a chain, clusters and teams in global memory."""
    rng = np.random.default_rng(n)
    v = np.arange(n)
    adj = np.stack([(v + s) % n for s in rng.permutation(n // 2 - 1)[:d] + 1], axis=1).astype(np.int32)   # one way round
    a = og.Anneal([og.Chain(adj, nodes=n, seed=k + 1, max_temp=50.0, min_temp=0.5, ncalcs=200) for k in range(count)])
    for _ in range(2):
        a.run(3)
        for k in range(count):
            x = a.state(k, graphs=True)
            assert x["status"] == 1 and x["steps"] == 0
            assert np.array_equal(x["adjacency"], adj) and np.array_equal(x["best_adjacency"], adj)
    a.close()


def test_a_cta_walks_several_chains(monkeypatch):
    """All of 700 chains, two or three to a CTA."""
    kw = dict(max_temp=50.0, min_temp=0.5, ncalcs=200)
    made = [og.Chain(general(60 + k % 5 * 12, 4, 1, k), nodes=60 + k % 5 * 12, seed=k, **kw) for k in range(700)]
    monkeypatch.setenv("ODP_GB300_ANNEAL_RESIDENT", "1")
    a = og.Anneal(made)
    monkeypatch.setenv("ODP_GB300_ANNEAL_RESIDENT", "0")
    b = og.Anneal(made)
    for steps in (1, 13):
        a.run(steps)
        b.run(steps)
        for k in range(len(made)):
            x, y = a.state(k, graphs=True), b.state(k, graphs=True)
            assert np.array_equal(x.pop("adjacency"), y.pop("adjacency")), (k, steps)
            assert np.array_equal(x.pop("best_adjacency"), y.pop("best_adjacency")), (k, steps)
            assert x == y, (k, steps)
    a.close()
    b.close()


def test_a_run_of_several_launches(monkeypatch):
    """More steps than a launch takes; only the last one leaves the state on the host."""
    kw = dict(max_temp=20.0, min_temp=0.1, ncalcs=2000)
    made = [og.Chain(general(n, 5, 1, n), nodes=n, seed=n, **kw) for n in (40, 64, 130)]
    monkeypatch.setenv("ODP_GB300_ANNEAL_RESIDENT", "1")
    a = og.Anneal(made)
    monkeypatch.setenv("ODP_GB300_ANNEAL_RESIDENT", "0")
    b = og.Anneal(made)
    for steps in (513, 512, 1100):
        a.run(steps)
        b.run(steps)
        for k in range(len(made)):
            x, y = a.state(k, graphs=True), b.state(k, graphs=True)
            assert np.array_equal(x.pop("adjacency"), y.pop("adjacency")), (k, steps)
            assert np.array_equal(x.pop("best_adjacency"), y.pop("best_adjacency")), (k, steps)
            assert x == y, (k, steps)
    a.close()
    b.close()
