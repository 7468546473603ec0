"""The kernels behind the lockstep ones, which larger graphs, schedule settings
and busy servers still take: the persistent engine with its pull kernel, and
the small-graph kernel at sizes where single graphs go to lockstep."""
import numpy as np
import pytest

import odp_gb300 as og
import oracle
from conftest import same

pytestmark = pytest.mark.gpu


def general(n, d, s=1, seed=1):
    return og.conv_edge2adjacency_general(n, og.generate_random_general(n, d, s, seed=seed), d, s)


def grid(w, h, d, length, s=1, seed=1):
    return og.conv_edge2adjacency_grid(w, h, og.generate_random_grid(w, h, d, length, s, seed=seed), d, s)


def graphs():
    rng = np.random.default_rng(9)
    irregular = rng.integers(0, 700, (700, 7)).astype(np.int32)
    nd = rng.integers(1, 8, 700).astype(np.int32)
    half = general(128, 4, seed=9)
    return [og.GraphSpec(general(1000, 12, seed=6), nodes=1000), og.GraphSpec(general(1000, 10, 4, 7), nodes=1000, symmetries=4),
            og.GraphSpec(irregular, nodes=700, num_degrees=nd), og.GraphSpec(np.concatenate([half, half + 128]), nodes=256),
            og.GraphSpec(general(4096, 24, seed=3), nodes=4096), og.GraphSpec(grid(30, 31, 6, 3), grid=True, width=30, height=31),
            og.GraphSpec(grid(40, 40, 4, 3, 4), grid=True, width=40, height=40, symmetries=4),
            og.GraphSpec(grid(160, 130, 4, 6), grid=True, width=160, height=130), og.GraphSpec(general(16, 3, seed=2), nodes=16)]


def wanted(g):
    return oracle.aspl(g.adjacency, nodes=g.nodes, num_degrees=g.num_degrees, symmetries=g.symmetries, grid=g.grid,
                       width=g.width, height=g.height)


def run_all(plans, path):
    """Each plan twice, with an out-of-range entry in between."""
    for specs in plans:
        want = [wanted(g) for g in specs]
        b = og.Batch(specs)
        assert b.path() == path
        for _ in range(2):
            assert all(same(x, y) for x, y in zip(b.run(), want)), [g.adjacency.shape for g in specs]
            bad = [g.adjacency.copy() for g in specs]
            bad[-1][0, 0] = bad[-1].size + 1000000
            with pytest.raises(og.ODPError) as e:
                b.run(bad)
            assert e.value.code == og.ERR_ADJACENCY
        b.close()


def test_engine_and_pull(monkeypatch):
    monkeypatch.setenv("ODP_GB300_SWEEP", "0")
    monkeypatch.setenv("ODP_GB300_SMALL_N", "0")
    g = graphs()
    run_all([[x] for x in g] + [g], "engine")


@pytest.mark.parametrize("env", ["ODP_GB300_SWEEP", "ODP_GB300_SMALL_CLUSTER"])
def test_small_kernel_past_the_line_to_lockstep(env, monkeypatch):
    plans = [[og.GraphSpec(general(3000, 16, seed=31), nodes=3000)], [og.GraphSpec(general(4096, 8, seed=32), nodes=4096)],
             [og.GraphSpec(grid(60, 61, 8, 4, seed=3), grid=True, width=60, height=61)]]
    for p in plans[:2]:
        b = og.Batch(p)
        assert b.path() == "lockstep" and b.kernel() == "small"
        b.close()
    monkeypatch.setenv(env, "0" if env == "ODP_GB300_SWEEP" else "8")
    run_all(plans, "small")


def test_calls_beside_a_busy_server():
    """They give the same results on the kernels they take then."""
    plans = [[x] for x in graphs()[4:8]] + [graphs()[:7]]      # the largest grid's bitsets exceed a team's
    want = [[wanted(g) for g in p] for p in plans]
    batches = [og.Batch(p) for p in plans]
    alone = [b.path() for b in batches]
    assert "lockstep" in alone and "teams" in alone
    srv = og.Server(lanes=2, max_nodes=160 * 130, memory_mb=512)
    handles = [srv.register(og.GraphSpec(grid(160, 130, 4, 6, seed=k), grid=True, width=160, height=130)) for k in range(4)]
    seen = set()
    for _ in range(6):
        ids = [srv.submit(h, []) for h in handles]
        for b, w in zip(batches, want):
            assert all(same(x, y) for x, y in zip(b.run(), w))
            seen.add(b.path())
        for r in ids:
            srv.wait(r)
        for b, w, path in zip(batches, want, alone):
            assert all(same(x, y) for x, y in zip(b.run(), w))
            assert b.path() == path
    assert "engine" in seen
    srv.close()
    for b in batches:
        b.close()
