"""Class-coded races of networks whose last Philox block is partly filled, and
of networks with members outside the classes (none, some or all components of
a block at a time), and lane groups of the largest networks: traces and
importance-sampling runs equal the CPU
oracle's bit for bit."""
import os
import tempfile

import numpy as np
import pytest

import oracle
from cusmc_b200 import api, netgen
from cusmc_b200 import proposal as P

pytestmark = pytest.mark.gpu


def _blob(w):
    with tempfile.NamedTemporaryFile("w", suffix=".xml", delete=False) as f:
        f.write(w.xml)
    try:
        return api.compile_model(f.name)
    finally:
        os.unlink(f.name)


NETS = {f"epidemic{n}": (lambda n=n: netgen.epidemic(n_agents=n, horizon=20, r_threshold=max(1, n // 3)))
        for n in (4, 5, 6, 7, 33, 99, 254, 255)}
NETS.update({f"mutex{n}": (lambda n=n: netgen.mutex(n, horizon=8)) for n in (4, 5, 6, 7, 33, 66)})


@pytest.mark.parametrize("name", sorted(NETS))
def test_class_coded_traces_match_the_oracle(name):
    w = NETS[name]()
    blob = _blob(w)
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=3000)
    m = 200
    _, want, _ = oracle.run(blob, q, 13, m, threads=0, digests=True, final_state=True)
    net = api.Network(blob)
    try:
        net.set_plan(4, 1, 1, 64)
        r, got = net.run_verify(q, 13, m)
        assert r.family == 4
    finally:
        net.close()
    for key in ("steps", "flags", "digests", "final_state"):
        assert np.array_equal(got[key], want[key]), key
    assert np.array_equal(got["values"].view(np.uint64), want["values"].view(np.uint64))


@pytest.mark.parametrize("name", sorted(n for n in NETS if n not in ("epidemic254", "mutex66")))
def test_weighted_runs_match_the_oracle(name):
    import torch
    w = NETS[name]()
    blob = _blob(w)
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=3000)
    prop = P.Proposal.init(3)
    prop.w3 = (np.random.default_rng(4).standard_normal(P.HID) * 0.1).astype(np.float32)
    params = prop.pack()
    m = 200
    cpu, _ = oracle.is_run(blob, q, params, 17, m, 40)
    net = api.Network(blob)
    try:
        P.set_inference(net, False)
        P.set_kernel(net, 5)
        logw = torch.zeros(m, dtype=torch.float64, device="cuda")
        steps = torch.zeros(m, dtype=torch.int32, device="cuda")
        r = P.is_run(net, q, params, 17, m, 40, logw=logw, steps=steps)
        assert r.family == 5
    finally:
        net.close()
    assert np.array_equal(steps.cpu().numpy().view(np.uint32), cpu["steps"])
    assert np.array_equal(logw.cpu().numpy().view(np.uint64), cpu["logw"].view(np.uint64))


@pytest.mark.parametrize("n_comps", [450, 500])
def test_lane_groups_of_networks_near_the_shared_memory_limit(n_comps):
    """The network, the variables and the slot masks of a 256-thread CTA's
    groups fit, their delay records do not: lane groups all the same."""
    w = netgen.random_network(8, n_comps=n_comps, horizon=1)
    blob = _blob(w)
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=300)
    _, want, _ = oracle.run(blob, q, 13, 40, threads=0, digests=True, final_state=True)
    net = api.Network(blob)
    try:
        for plan in (None, (0, 32, 16, 256), (0, 32, 16, 64)):
            if plan:
                net.set_plan(*plan)
            r, got = net.run_verify(q, 13, 40)
            assert (r.family, r.lanes_per_run) == (0, 32)
            for key in ("steps", "flags", "digests", "final_state"):
                assert np.array_equal(got[key], want[key]), (plan, key)
    finally:
        net.close()


def test_networks_beyond_shared_memory_run_a_warp_per_run():
    w = max(netgen.batch_networks(64, base_seed=1000), key=lambda w: len(w.xml))
    blob = _blob(w)
    assert len(blob) > 232_448
    q = api.variable_query(w.var_id, 1, threshold=w.threshold, is_max=True, max_steps=300)
    _, want, _ = oracle.run(blob, q, 13, 40, threads=0, digests=True, final_state=True)
    net = api.Network(blob)
    try:
        for plan, lanes in ((None, 32), ((2, 1, 1, 128), 1)):
            if plan:
                net.set_plan(*plan)
            r, got = net.run_verify(q, 13, 40)
            assert (r.family, r.lanes_per_run) == (2, lanes)
            for key in ("steps", "flags", "digests", "final_state"):
                assert np.array_equal(got[key], want[key]), (plan, key)
            assert np.array_equal(got["values"].view(np.uint64), want["values"].view(np.uint64))
    finally:
        net.close()


@pytest.mark.parametrize("workload,first,variables,plan,family", [
    # class-coded CTAs of 32 threads: the keys of 128 fit, or only those of 32
    (lambda: netgen.epidemic(n_agents=40, horizon=20, r_threshold=10), "int S = 39;", 1500, (4, 1, 1, 32), 4),
    (lambda: netgen.epidemic(n_agents=40, horizon=20, r_threshold=10), "int S = 39;", 1600, (4, 1, 1, 32), 1),
    # one warp per run: its records fit, or only its variables and slot masks
    (lambda: netgen.mutex(300, horizon=3), "int id = 0;", 10_000, (0, 32, 16, 32), 0),
    (lambda: netgen.mutex(300, horizon=3), "int id = 0;", 11_016, (0, 32, 16, 32), 1),
])
def test_plans_at_the_shared_memory_limit_report_what_runs(workload, first, variables, plan, family):
    w = workload()
    w.xml = w.xml.replace(first, first + "\n" + "\n".join(f"int u{i} = {i % 9};" for i in range(variables)), 1)
    blob = _blob(w)
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=300)
    _, want, _ = oracle.run(blob, q, 13, 40, threads=0, digests=True, final_state=True)
    net = api.Network(blob)
    try:
        net.set_plan(*plan)
        r, got = net.run_verify(q, 13, 40)
        assert r.family == family and r.lanes_per_run == net.plan()[0]
    finally:
        net.close()
    for key in ("steps", "flags", "digests", "final_state"):
        assert np.array_equal(got[key], want[key]), key
