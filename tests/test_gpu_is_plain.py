"""Importance sampling one warp per run on networks without invariants: runs,
log-weights and replayed rows equal the CPU oracle's bit for bit where what
the kernel keeps between steps goes stale in different ways: component
counts that leave the last Philox block partly filled, more than one block
per lane, zero-delay locations, clocks (in guards, in rates, as the clock
feature), broadcast receivers, CTAs of one to eight warps."""
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


def _clocked(n, rate):
    """n clocked automata: an exponential location whose edge waits for the
    clock, an urgent one, and one whose edge wakes the others."""
    d = netgen._Doc("int v0 = 0;\nint v1 = 1;\nint v2 = 0;\nint v3 = 0;\nbroadcast chan go;")
    for c in range(n):
        a, u, b = d.new_id(), d.new_id(), d.new_id()
        d.template(f"K{c}", "clock x;", [(a, "a", [("exponentialrate", rate)]), (u, "u", []),
                                         (b, "b", [("exponentialrate", "1.25")])],
                   a, [(a, u, [("guard", "x >= 1"), ("assignment", "v0 = v0 + 1")]),
                       (u, b, [("assignment", "v2 = v2 + 1, x = 0")]),
                       (b, a, [("synchronisation", "go!"), ("assignment", "v1 = v1 + 1")]),
                       (b, a, [("synchronisation", "go?"), ("assignment", "v3 = v3 + 1")])])
    xml = d.finish().replace('<name>u</name>', '<name>u</name><urgent/>')
    return netgen.Workload("clocked", xml, var_id=0, threshold=5, horizon=8, runs=100)


CASES = {
    "epidemic3": (lambda: netgen.epidemic(n_agents=3, horizon=20, r_threshold=2), -1),
    "epidemic37": (lambda: netgen.epidemic(n_agents=37, horizon=30, r_threshold=10), -1),
    "epidemic135": (lambda: netgen.epidemic(n_agents=135, horizon=15, r_threshold=10), -1),
    "clocked_literal": (lambda: _clocked(5, "0.7"), 4),
    "clocked_rate": (lambda: _clocked(6, "0.4 + 0.3 * v1"), -1),
    "clocked_clock_rate": (lambda: _clocked(6, "0.2 + x * 0.5"), 5),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_runs_and_rows_match_the_oracle(name):
    import torch
    make, clock_var = CASES[name]
    w = make()
    blob = _blob(w)
    q = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True, max_steps=4000)
    prop = P.Proposal.init(3)
    prop.w3 = (np.random.default_rng(4).standard_normal(P.HID) * 0.1).astype(np.float32)
    params = prop.pack()
    info = api.blob_info(blob)
    feats = P.pack_features(info["n_vars"], info["n_comps"], clock_var=clock_var)
    net = api.Network(blob)
    dev = torch.device("cuda")
    try:
        P.set_inference(net, False)
        P.set_kernel(net, 3)
        P.set_features(net, [i if i < info["n_vars"] else -1 for i in range(4)],
                       [float(np.float32(1.0) / np.float32(info["n_comps"]))] * 4, clock_var)
        for n in (5, 200, 700):
            flags = torch.zeros(n, dtype=torch.uint8, device=dev)
            logw = torch.zeros(n, dtype=torch.float64, device=dev)
            values = torch.zeros(n, dtype=torch.float64, device=dev)
            steps = torch.zeros(n, dtype=torch.int32, device=dev)
            P.is_run(net, q, params, 17, n, 40, flags=flags, logw=logw, values=values, steps=steps)
            cpu, _ = oracle.is_run(blob, q, params, 17, n, 40, features=feats)
            assert np.array_equal(steps.cpu().numpy().view(np.uint32), cpu["steps"])
            assert np.array_equal(flags.cpu().numpy(), cpu["flags"])
            assert np.array_equal(values.cpu().numpy().view(np.uint64), cpu["values"].view(np.uint64))
            assert np.array_equal(logw.cpu().numpy().view(np.uint64), cpu["logw"].view(np.uint64))
        runs = np.array([0, 3, 9, 150, 699], dtype=np.uint64)
        wts = np.array([0.1, 0.4, 0.2, 0.05, 0.25], dtype=np.float32)
        want = oracle.is_trace(blob, q, params, 17, runs, wts, 40, features=feats)
        st = cpu["steps"][runs.astype(np.int64)].astype(np.int64)
        offs = np.concatenate([[0], np.cumsum(4 * st)[:-1]]).astype(np.uint64)
        rows = torch.zeros(len(want) * P.ROW_BYTES, dtype=torch.uint8, device=dev)
        P.is_trace(net, q, params, 17, torch.from_numpy(runs.view(np.int64)).to(dev), torch.from_numpy(wts).to(dev),
                   torch.from_numpy(offs.view(np.int64)).to(dev), rows, 40)
        assert rows.cpu().numpy().tobytes() == want.tobytes()
    finally:
        net.close()
