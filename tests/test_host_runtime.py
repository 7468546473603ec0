"""The host runtime (plans, batches, servers, annealing) over a CUDA layer
without a GPU (c/fake_gpu.c): what it does when launches fail, and which
kernels it launches."""
import ctypes
import os
import subprocess
import time

import numpy as np
import pytest

import odp_gb300 as og
from conftest import ROOT
from odp_gb300 import build

KINDS = ("engine", "small", "sweep", "team", "resident", "step", "pull")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.run(["gcc", "-O1", "-std=gnu11", "-fPIC", "-shared", "-w", "-I", build.INCLUDE, "-I", build.CSRC, "-o", so,
                    os.path.join(ROOT, "tests", "c", "fake_gpu.c")] +
                   [os.path.join(build.CSRC, f) for f in build.C_SOURCES] + ["-lm", "-lpthread"], check=True)
    return so


class Fake:
    """The fake layer's counters and switches, in the loaded library."""

    def __init__(self, lib):
        object.__setattr__(self, "lib", lib)
        self.counts = 0

    def __setattr__(self, name, value):
        if name == "counts":
            (ctypes.c_int * len(KINDS)).in_dll(self.lib, "fake_launches")[:] = [value] * len(KINDS)
        else:
            ctypes.c_int.in_dll(self.lib, "fake_" + name).value = value

    def __getattr__(self, name):
        if name == "counts":
            return {k: v for k, v in zip(KINDS, (ctypes.c_int * len(KINDS)).in_dll(self.lib, "fake_launches")) if v}
        return ctypes.c_int.in_dll(self.lib, "fake_" + name).value


@pytest.fixture
def fake(library, monkeypatch):
    """The package on the fake layer, without CUDA graphs."""
    monkeypatch.setattr(og, "LIB_PATH", library)
    monkeypatch.setattr(og, "_lib", None)
    monkeypatch.setenv("ODP_GB300_GRAPH", "0")
    f = Fake(og.load())
    yield f
    f.abort_at = f.late_at = f.pending = f.pending_from = 0


def ring(n, d=4):
    v = np.arange(n)
    return np.stack([(v + 1 + k) % n for k in range(d)], axis=1).astype(np.int32)


def launched(fake, kind):
    """Waits for the server's thread to launch its batch."""
    stop = time.monotonic() + 30
    while kind not in fake.counts and time.monotonic() < stop:
        time.sleep(1e-4)
    assert kind in fake.counts


def timed_out(call):
    with pytest.raises(og.ODPError) as e:
        call()
    return e.value.code == og.ERR_TIMEOUT


def plans():
    return {"sweep": [og.GraphSpec(ring(6000), nodes=6000)],
            "team": [og.GraphSpec(ring(n), nodes=n) for n in (6000, 9000, 700)]}


@pytest.mark.parametrize("kind", ["sweep", "team"])
def test_a_wait_that_ran_out_fails_its_own_call_only(fake, kind):
    """In a run, and in a timed launch after a warm one."""
    b = og.Batch(plans()[kind])
    b.run()
    assert fake.counts == {kind: 1}
    fake.abort_at = fake.total + 1
    assert timed_out(b.run)
    b.run()
    fake.abort_at = fake.total + 3
    assert timed_out(lambda: b.time(4))
    b.run()
    b.close()


def test_a_wait_that_ran_out_behind_the_last_record_is_no_failure(fake):
    """All records of a launch are its results, also when a CTA that had nothing
    left to do gave up its wait for the last barrier, before or after the host
    looked."""
    b = og.Batch(plans()["sweep"])
    want = b.run()
    fake.late_at = fake.total + 1
    assert b.run() == want
    assert b.run() == want
    b.close()


def served(server, graphs):
    handles = [server.register(g) for g in graphs]
    for _ in range(2):
        for r in [server.submit(h, []) for h in handles]:
            server.wait(r)


def test_a_server_with_graphs_for_the_engine_keeps_all_on_it(fake):
    """Team batches take SMs from an engine batch that starts beside them."""
    general = [og.GraphSpec(ring(n), nodes=n) for n in (300, 2000)]
    grid = og.GraphSpec(ring(400), grid=True, width=20, height=20)
    srv = og.Server(max_nodes=2000, memory_mb=64)
    served(srv, general)
    assert set(fake.counts) == {"team"}
    fake.counts = 0
    served(srv, [grid])
    served(srv, general)
    assert set(fake.counts) == {"engine"}
    srv.close()


def test_choosing_teams_is_linear_in_the_graphs(fake):
    """Each graph's fit is looked at once per size of team, whatever the shares
    and teams that are tried."""
    specs = [og.GraphSpec(np.zeros((64 * (k % 50) + 300, 6), np.int32), nodes=64 * (k % 50) + 300) for k in range(700)]
    asked = fake.asked
    b = og.Batch(specs)
    assert fake.asked - asked <= 12 * len(specs)
    b.close()


@pytest.mark.parametrize("kind", ["sweep", "team"])
def test_calls_beside_a_servers_long_batches_take_no_cooperative_launch(fake, kind):
    """Such a launch waits for the whole GPU.  With the server idle again, or
    closed with its batch in flight, the call takes it again."""
    nd = np.full(6000, 4, np.int32)
    nd[5] = 3
    specs = plans()[kind]
    specs[0] = og.GraphSpec(ring(6000), nodes=6000, num_degrees=nd)
    b = og.Batch(specs)
    nd[:] = 0                                            # the plan keeps its own
    want = b.run()
    assert fake.counts == {kind: 1}
    for closed in (0, 1):
        srv = og.Server(max_nodes=2000, memory_mb=64)
        h = srv.register(og.GraphSpec(ring(400), grid=True, width=20, height=20))
        fake.pending = 1
        r = srv.submit(h, [])
        launched(fake, "engine")
        fake.counts = 0
        assert b.run() == want and b.run() == want
        assert set(fake.counts) == {"engine", "pull"} and fake.counts["engine"] == 2
        assert len(b.job_levels()) == b.info(0)["njobs"] and (b.job_levels() == 1).all()
        fake.pending = 0
        if not closed:
            srv.wait(r)
        else:
            fake.pending = 1
            r = srv.submit(h, [])
        srv.close()
        fake.pending = fake.counts = 0
        assert b.run() == want and fake.counts == {kind: 1}
    b.close()


def test_calls_beside_a_servers_short_team_batches_stay_in_lockstep(fake):
    b = og.Batch(plans()["sweep"])
    srv = og.Server(max_nodes=2000, memory_mb=64)
    h = srv.register(og.GraphSpec(ring(2000), nodes=2000))
    fake.abort_at = fake.total + 1                       # no records: in flight until its event is complete
    fake.pending = 1
    r = srv.submit(h, [])
    launched(fake, "team")
    fake.counts = fake.abort_at = 0
    b.run()
    assert fake.counts == {"sweep": 1}
    fake.pending = 0
    with pytest.raises(og.ODPError):
        srv.wait(r)
    srv.close()
    b.close()


def test_timing_after_a_call_beside_a_server_reads_that_calls_arrays(fake):
    """ODPX_Batch_time without arrays times the last run's."""
    b = og.Batch(plans()["sweep"])
    first, second = ring(6000), ring(6000, 4)[:, ::-1].copy()
    b.run([first])
    srv = og.Server(max_nodes=2000, memory_mb=64)
    h = srv.register(og.GraphSpec(ring(400), grid=True, width=20, height=20))
    fake.pending = 1
    r = srv.submit(h, [])
    launched(fake, "engine")
    fake.counts = 0
    b.run([second])
    assert fake.counts["engine"] == 1 and "sweep" not in fake.counts
    fake.pending = 0
    srv.wait(r)
    srv.close()
    ms = ctypes.c_float()
    assert og.load().ODPX_Batch_time_mode(b._h, None, 2, 0, 0, ctypes.byref(ms)) == 0
    assert ctypes.c_void_p.in_dll(fake.lib, "fake_adjacency").value == second.ctypes.data
    b.close()


@pytest.mark.parametrize("graphs,env,path", [
    ([(300, 4)], {}, "small"), ([(4000, 24)], {}, "lockstep"), ([(4000, 24)], {"ODP_GB300_SWEEP": "0"}, "engine"),
    ([(2000, 8)], {}, "lockstep"), ([(2000, 8)], {"ODP_GB300_SWEEP": "0"}, "small"), ([(2000, 8)], {"ODP_GB300_SMALL_CLUSTER": "8"}, "small"),
    ([(6000, 4), (700, 4)], {}, "teams"), ([(6000, 4), (700, 4)], {"ODP_GB300_SWEEP": "0"}, "engine"),
    ([(6000, 4)], {"ODP_GB300_SLOTS": "3"}, "engine")])
def test_the_path_names_the_kernels_that_run(fake, graphs, env, path, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    b = og.Batch([og.GraphSpec(ring(n, d), nodes=n) for n, d in graphs])
    assert b.path() == path
    fake.counts = 0
    b.run()
    assert set(fake.counts) - {"pull"} == {{"lockstep": "sweep", "teams": "team"}.get(path, path)}
    assert b.path() == path
    b.close()


@pytest.mark.parametrize("n,s,d,path", [(262144, 4096, 8, "engine"), (262144, 1024, 8, "lockstep"), (130000, 1300, 8, "lockstep"), (130100, 1301, 8, "engine"),
                                        (160000, 1600, 4, "lockstep"), (800000, 800, 6, "engine"), (800000, 500, 6, "lockstep"), (420000, 420, 6, "lockstep")])
def test_graphs_of_many_rows_and_few_sources_stay_on_the_engine(fake, n, s, d, path):
    """Both sides of the lines where the engine is the faster one."""
    adj = np.zeros((n // s, d), np.int32)
    b = og.Batch([og.GraphSpec(adj, nodes=n, symmetries=s)])
    assert b.path() == path
    b.run()
    b.close()


@pytest.mark.parametrize("graphs,path", [
    ([(20000, 100, 8)] * 40, "engine"), ([(8000, 4, 8)] * 50, "engine"), ([(8000, 4, 8)] * 10, "teams"), ([(20000, 100, 8)] * 3, "teams"),
    ([(2000, 1, 8)] * 20 + [(200000, 2000, 8)] * 3, "engine"), ([(8000, 1, 8)] * 60 + [(8000, 4, 8)] * 30, "teams")])
def test_batches_that_lose_on_teams_stay_on_the_engine(fake, graphs, path):
    """Graphs of many rows a source, alone and among others."""
    b = og.Batch([og.GraphSpec(np.zeros((n // s, d), np.int32), nodes=n, symmetries=s) for n, s, d in graphs])
    assert b.path() == path
    b.close()


@pytest.mark.parametrize("w,h,d,s,count,path", [(150, 150, 40, 1, 1, "lockstep"), (170, 170, 40, 1, 1, "engine"), (170, 170, 32, 1, 1, "lockstep"),
                                                (256, 256, 36, 4, 1, "lockstep"), (256, 256, 36, 2, 1, "engine"), (54, 55, 36, 1, 40, "teams"),
                                                (56, 56, 36, 1, 40, "engine"), (56, 56, 32, 1, 40, "teams")])
def test_dense_grids_that_lose_in_lockstep_stay_on_the_engine(fake, w, h, d, s, count, path):
    """Both sides of the lines, and grids whose changes are tracked."""
    adj = np.zeros((w * h // s, d), np.int32)
    b = og.Batch([og.GraphSpec(adj, grid=True, width=w, height=h, symmetries=s)] * count)
    assert b.path() == path
    b.close()


@pytest.mark.parametrize("n,s,kernel", [(8000, 125, "engine"), (4000, 62, "team"), (20000, 100, "engine"), (20000, 10, "team"), (2000, 4, "team")])
def test_served_graphs_of_many_rows_a_source_stay_on_the_engine(fake, n, s, kernel):
    n = n // s * s
    srv = og.Server(max_nodes=n, memory_mb=512)
    served(srv, [og.GraphSpec(np.zeros((n // s, 8), np.int32), nodes=n, symmetries=s)])
    assert set(fake.counts) == {kernel}
    srv.close()


def test_long_calls_wait_for_team_batches(fake):
    """Behind long team batches a short call goes to the other kernels, a long one
    stays in lockstep."""
    plans = [og.Batch([g]) for g in (og.GraphSpec(ring(4096, 24), nodes=4096), og.GraphSpec(ring(97 * 103, 6), grid=True, width=97, height=103),
                                     og.GraphSpec(ring(30000, 4), nodes=30000))]
    srv = og.Server(lanes=1, max_nodes=8192, memory_mb=512)
    handles = [srv.register(og.GraphSpec(ring(8192, 8), nodes=8192)) for _ in range(17)]
    fake.pending = 1
    fake.abort_at = fake.total + 1                       # a batch of one, in flight without records
    ids = [srv.submit(handles[0], [])]
    launched(fake, "team")
    ids += [srv.submit(h, []) for h in handles[1:]]      # these wait for the lane, and then make one batch
    for b in plans:
        b.run()
    assert [b.path() for b in plans] == ["lockstep"] * 3
    fake.counts = 0
    fake.abort_at = fake.pending_from = fake.total + 1   # which stays in flight as well
    fake.pending = 0
    launched(fake, "team")
    for b in plans:
        b.run()
    assert [b.path() for b in plans] == ["engine", "lockstep", "lockstep"]
    fake.pending_from = 0
    for r in ids:
        assert timed_out(lambda: srv.wait(r))
    srv.close()
    for b in plans:
        b.run()
        assert b.path() == "lockstep"
        b.close()
