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


def random_spec(rng, n_hi):
    kind = rng.integers(0, 5)
    if kind == 0:
        w, h = int(rng.integers(2, 31)), int(rng.integers(2, 31))
        s = int(rng.choice([1, 2])) if w % 2 == 0 else 1
        d = int(rng.integers(1, 40))
        base = w * h // s
        cells = np.arange(base)
        step = rng.integers(-3, 4, (base, d))
        adj = np.clip(cells[:, None] + step, 0, w * h - 1).astype(np.int32)
        return og.GraphSpec(adj, grid=True, width=w, height=h, symmetries=s)
    s = int(rng.choice([1, 1, 2, 3, 7]))
    base = int(np.exp(rng.uniform(0, np.log(n_hi // s)))) + (1 if kind == 1 else 0)
    n, d = base * s, int(rng.integers(1, 13) if kind else rng.integers(60, 90))
    adj = np.stack([rng.permutation(base) + base * rng.integers(0, s, base) for _ in range(d)], axis=1).astype(np.int32)
    nd = rng.integers(0, d + 1, base).astype(np.int32) if kind == 2 else None
    return og.GraphSpec(adj, nodes=n, symmetries=s, num_degrees=nd)


@pytest.mark.parametrize("count,n_hi", [(2, 3000), (3, 40), (17, 6000), (60, 2000), (400, 300)])
def test_batches(count, n_hi):
    """Teams of every size: uneven graphs, two calls with other arrays, an
    out-of-range entry and a wait that runs out in between."""
    rng = np.random.default_rng(count)
    specs = [random_spec(rng, n_hi) for _ in range(count)]
    want = [oracle.aspl(g.adjacency, nodes=0 if g.grid else g.nodes, num_degrees=g.num_degrees,
                        symmetries=g.symmetries, grid=g.grid, width=g.width, height=g.height) for g in specs]
    b = og.Batch(specs)
    b.set_wait_limit(5 * 10 ** 9)
    for got in (b.run(), b.run()):
        for k, (x, y) in enumerate(zip(got, want)):
            assert same(x, y), (k, specs[k].grid, specs[k].nodes, specs[k].adjacency.shape, x, y)
    k = int(np.argmax([g.adjacency.size if g.num_degrees is None else 0 for g in specs]))
    bad = [g.adjacency for g in specs]
    bad[k] = bad[k].copy()
    bad[k][-1, -1] = specs[k].nodes
    with pytest.raises(og.ODPError) as e:
        b.run(bad)
    assert e.value.code == og.ERR_ADJACENCY
    turned = [np.ascontiguousarray(g.adjacency[:, ::-1]) if g.num_degrees is None else g.adjacency for g in specs]
    assert all(same(x, y) for x, y in zip(b.run(turned), want))
    b.close()


@pytest.mark.parametrize("n,d,kind", [(2048, 3, "undirected"), (5000, 4, "directed"), (8600, 3, "undirected"),
                                      (8601, 3, "directed"), (6000, 6, "irregular"), (7000, 2, "rings"),
                                      (5001, 5, "halves"), (20000, 5, "undirected"), (33000, 9, "directed"),
                                      (70000, 3, "halves")])
def test_levels_from_the_lists(n, d, kind, monkeypatch):
    """Three and more levels from the neighbour lists: undirected and directed
    lists (whose trees fill the queue), rows of several lengths, levels that end
    early (rings of 40, components), one group and several."""
    rng = np.random.default_rng(n)
    nd = None
    if kind == "undirected":
        adj = og.conv_edge2adjacency_general(n, og.generate_random_general(n, d - (n * d) % 2, seed=n), d - (n * d) % 2)
    elif kind == "rings":
        v = np.arange(n)
        adj = np.stack([v // 40 * 40 + (v + 1) % 40, v // 40 * 40 + (v + 39) % 40], axis=1).astype(np.int32)
        adj = np.minimum(adj, n - 1)
    else:
        half = n // 2 if kind == "halves" else n
        adj = np.stack([np.concatenate([rng.permutation(half), half + rng.permutation(n - half)]) for _ in range(d)],
                       axis=1).astype(np.int32)
        if kind == "irregular":
            nd = rng.integers(d - 2, d + 1, n).astype(np.int32)
    b = og.Batch([og.GraphSpec(adj, nodes=n, num_degrees=nd)])
    got = b.run()[0]
    b.close()
    if n <= 9000:
        assert same(got, oracle.aspl(adj, nodes=n, num_degrees=nd))
    monkeypatch.setenv("ODP_GB300_SWEEP", "0")
    b = og.Batch([og.GraphSpec(adj, nodes=n, num_degrees=nd)])
    assert same(got, b.run()[0])
    b.close()


@pytest.mark.parametrize("w,h,d,length", [(61, 47, 7, 4), (100, 90, 8, 4), (40, 33, 14, 5), (45, 40, 20, 6), (33, 30, 32, 8)])
def test_grids_with_eight_neighbours_in_flight(w, h, d, length):
    d -= (w * h * d) % 2
    adjs = [og.conv_edge2adjacency_grid(w, h, og.generate_random_grid(w, h, d, length, 1, seed=k), d, 1) for k in (3, 4)]
    check(og.GraphSpec(adjs[0], grid=True, width=w, height=h), adjs)


@pytest.mark.parametrize("w,h,d,length", [(139, 140, 4, 5), (140, 140, 6, 6), (100, 230, 3, 6)])
def test_grids_of_three_ctas_per_sm(w, h, d, length, monkeypatch):
    """On both sides of the line where a level takes a second round."""
    adj = og.conv_edge2adjacency_grid(w, h, og.generate_random_grid(w, h, d, length, 1, seed=5), d, 1)
    b = og.Batch([og.GraphSpec(adj, grid=True, width=w, height=h)])
    got = b.run()[0]
    b.close()
    monkeypatch.setenv("ODP_GB300_SWEEP", "0")
    b = og.Batch([og.GraphSpec(adj, grid=True, width=w, height=h)])
    assert same(got, b.run()[0])
    b.close()


@pytest.mark.parametrize("kind", ["at once", "two phases", "tracking", "teams"])
def test_chunk_counts_meet_the_barrier(kind, monkeypatch):
    """Every lane of a CTA's first warp adds the counts of a chunk of its own
    and one lane arrives for all of them: graphs of several chunks per barrier,
    launched often, against the persistent engine."""
    rng = np.random.default_rng(11)

    def lists(n, d):
        return np.stack([rng.permutation(n) for _ in range(d)], axis=1).astype(np.int32)

    if kind == "tracking":
        w, h = 150, 131
        adj = og.conv_edge2adjacency_grid(w, h, og.generate_random_grid(w, h, 6, 6, 1, seed=9), 6, 1)
        specs = [og.GraphSpec(adj, grid=True, width=w, height=h)]
    elif kind == "teams":
        specs = [og.GraphSpec(lists(n, 7), nodes=n) for n in (16000, 9000, 12289, 8193, 5000)]
    else:
        n = 16000 if kind == "at once" else 40000
        specs = [og.GraphSpec(lists(n, 6), nodes=n)]
    b = og.Batch(specs)
    b.set_wait_limit(5 * 10 ** 9)
    got = [b.run() for _ in range(40)]
    b.close()
    monkeypatch.setenv("ODP_GB300_SWEEP", "0")
    b = og.Batch(specs)
    want = b.run()
    b.close()
    for run in got:
        assert all(same(x, y) for x, y in zip(run, want))


@pytest.mark.parametrize("count,n_hi", [(2, 3000), (17, 6000), (60, 2000)])
def test_batches_after_a_wait_that_runs_out(count, n_hi):
    """The teams give up their waits for one another, and the plan's next runs
    start from clean counters."""
    rng = np.random.default_rng(count + 1)
    specs = [random_spec(rng, n_hi) for _ in range(count)]
    b = og.Batch(specs)
    b.set_wait_limit(5 * 10 ** 9)
    want = b.run()
    for _ in range(2):
        b.set_wait_limit(1)
        with pytest.raises(og.ODPError) as e:
            b.run()
        assert e.value.code == og.ERR_TIMEOUT
        with pytest.raises(og.ODPError) as e:
            b.time(3)
        assert e.value.code == og.ERR_TIMEOUT
        b.set_wait_limit(5 * 10 ** 9)
        for _ in range(2):
            assert all(same(x, y) for x, y in zip(b.run(), want))
    b.close()


def test_batches_of_arrays_anywhere():
    """Every page of the arrays is asked for before the graphs are taken: arrays
    off 16-byte boundaries, ending with a page and a word behind one, new ones on
    each run, and one without entries."""
    import mmap
    rng = np.random.default_rng(21)
    page = mmap.PAGESIZE // 4
    shapes = [(2048, 8), (page // 4, 4), (page // 4 + 1, 4), (5000, 13), (97, 5), (100, 0), (6001, 11)]
    want = None
    for run in range(3):
        arrays, keep = [], []
        for n, d in shapes:
            m = mmap.mmap(-1, (n * d * 4 // mmap.PAGESIZE + 2) * mmap.PAGESIZE)
            keep.append(m)
            at = len(m) - 4 * n * d if run == 0 else 4 * run       # the last entries of the mapping, then odd offsets
            a = np.frombuffer(m, dtype=np.int32, count=n * d, offset=at).reshape(n, d)
            if want is None:
                a[:] = np.stack([rng.permutation(n) for _ in range(d)], axis=1) if d else 0
            else:
                a[:] = first[len(arrays)]
            arrays.append(a)
        if want is None:
            first = [a.copy() for a in arrays]
            want = [oracle.aspl(a, nodes=n) if d else (2**31 - 1, 2**63 - 1, float(np.finfo(np.float64).max))
                    for a, (n, d) in zip(arrays, shapes)]
            b = og.Batch([og.GraphSpec(a, nodes=n) for a, (n, d) in zip(first, shapes)])
        assert all(same(x, y) for x, y in zip(b.run(arrays), want)), run
    b.close()
