"""The launch plan is chosen by the number of runs (one thread per run, or a
group of 2 to 32 lanes per run with one to sixteen components per lane); a
run's results do not depend on it.

Each network is run at launch sizes on both sides of every choice, and the
first runs of each launch are compared bit for bit with the CPU oracle:
component counts at the edges of the lane shares (1, 2, 4, 5, 32, 33, 63
components), classes with and without other locations, invariants, clocks,
broadcast receivers, a location query.  Every lane-group shape is also run
through csmc_run_verify's traces.
"""
import os
import tempfile

import numpy as np
import pytest

import oracle
from cusmc_b200 import api, netgen

pytestmark = pytest.mark.gpu


def _blob(w, loc=""):
    with tempfile.NamedTemporaryFile("w", suffix=".xml", delete=False) as f:
        f.write(w.xml)
    try:
        return api.compile_model(f.name, loc, bool(loc))
    finally:
        os.unlink(f.name)


NETS = {
    "random1": lambda: netgen.random_network(3, n_comps=1, horizon=30),
    "random2": lambda: netgen.random_network(4, n_comps=2, horizon=30),
    "random5": lambda: netgen.random_network(5, n_comps=5, horizon=20),
    "random33": lambda: netgen.random_network(6, n_comps=33, horizon=6),
    "epidemic4": lambda: netgen.epidemic(n_agents=4, horizon=20, r_threshold=2),
    "epidemic63": lambda: netgen.epidemic(n_agents=63, horizon=12, r_threshold=20),
    "mutex32": lambda: netgen.mutex(32, horizon=6),
}


@pytest.mark.parametrize("name", sorted(NETS))
def test_every_launch_size_gives_the_oracle_runs(name):
    import torch
    w = NETS[name]()
    blob = _blob(w)
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=100_000)
    m = 200
    _, want, _ = oracle.run(blob, q, 77, m, threads=0)
    net = api.Network(blob)
    shapes = set()
    try:
        for n in (1, m, 5_000, 11_003, 24_000, 70_001):
            flags = torch.zeros(n, dtype=torch.uint8, device="cuda")
            values = torch.zeros(n, dtype=torch.float64, device="cuda")
            steps = torch.zeros(n, dtype=torch.int32, device="cuda")
            r = net.run(q, 77, n, flags=flags, values=values, steps=steps)
            shapes.add((r.family, r.lanes_per_run, r.comps_per_lane))
            k = min(n, m)
            assert np.array_equal(steps.cpu().numpy().view(np.uint32)[:k], want["steps"][:k])
            assert np.array_equal(flags.cpu().numpy()[:k], want["flags"][:k])
            assert np.array_equal(values.cpu().numpy()[:k], want["values"][:k])
            assert r.hits == int(flags.sum()) and r.steps == int(steps.to(torch.int64).sum())
    finally:
        net.close()
    # (up to two components one thread per run is taken at every size)
    assert len(shapes) >= (1 if name in ("random1", "random2") else 2), shapes


def test_location_query_at_small_and_large_launches():
    w = netgen.epidemic(n_agents=10, horizon=30)
    blob = _blob(w, "Agent3.R")
    q = api.location_query(w.horizon)
    _, want, _ = oracle.run(blob, q, 5, 400, threads=0)
    for n in (400, 90_000):
        _, flags, _, steps = api.run_host(blob, q, 5, n, want_steps=True)
        assert np.array_equal(flags[:400], want["flags"]) and np.array_equal(steps[:400], want["steps"])


@pytest.mark.parametrize("g,k,net", [
    (32, 1, "random2"), (16, 2, "mutex32"), (2, 4, "random5"), (4, 4, "mutex13"), (8, 4, "mutex32"), (16, 4, "epidemic63"), (4, 8, "mutex32"),
    (8, 8, "epidemic63"), (16, 8, "epidemic100"), (8, 16, "epidemic100"), (16, 16, "mutex130"), (32, 16, "random300"),
])
def test_lane_group_shapes_give_the_oracle_traces(g, k, net):
    make = dict(NETS, mutex13=lambda: netgen.mutex(13, horizon=20),
                epidemic100=lambda: netgen.epidemic(horizon=10), mutex130=lambda: netgen.mutex(130, horizon=3),
                random300=lambda: netgen.random_network(8, n_comps=300, horizon=2))
    w = make[net]()
    blob = _blob(w)
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=100_000)
    h = api.Network(blob)
    try:
        h.set_plan(0, g, k, 64)
        r, got = h.run_verify(q, 9, 300)
        assert (r.family, r.lanes_per_run, r.comps_per_lane) == (0, g, k)
    finally:
        h.close()
    _, want, _ = oracle.run(blob, q, 9, 300, threads=0, digests=True, final_state=True)
    for key in ("steps", "flags", "digests", "final_state"):
        assert np.array_equal(got[key], want[key]), key
    assert np.array_equal(got["values"].view(np.uint64), want["values"].view(np.uint64))


def test_autotuner_keeps_a_default_that_is_the_fastest():
    """8 components, 100 runs: one warp per run, 1.6 times faster than any
    fixed plan the autotuner tries.  The handle keeps choosing by the number
    of runs, also after a plan was set."""
    w = netgen.random_network(0, horizon=100)
    net = api.Network(_blob(w))
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=100_000)
    try:
        before = [net.run(q, 3, n) for n in (100, 70_001)]
        for plan in (None, (1, 1, 1, 128)):
            if plan:
                net.set_plan(*plan)
            best = net.autotune(q, 3, 100)
            assert (best.family, best.lanes_per_run) == (0, 32)
            for n, b in zip((100, 70_001), before):
                r = net.run(q, 3, n)
                assert (r.family, r.lanes_per_run, r.comps_per_lane) == (b.family, b.lanes_per_run, b.comps_per_lane)
                assert (r.hits, r.steps, r.sum) == (b.hits, b.steps, b.sum)
    finally:
        net.close()
