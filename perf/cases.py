"""Workloads of the model checker that are worth timing, through its public
Python entry points.

What a user does with this library, and the cases that stand for it:

* one question about one model: `api.run_host` (what the CLI and `api.smc`
  call: a packed network in, per-run flags and values out on the host) and
  `Network.run` (the same with the network resident and the results left on
  the device), from a quick look with a hundred runs to a tight estimate with
  a million, on networks of two automata up to a few hundred;
* many models at once: `api.Batch`, one launch for a list of (network, query)
  jobs of uneven size;
* rare events: runs under a proposal network (`proposal.is_run`), the replay
  of a training round's elite runs into training rows with the merge of equal
  rows (`proposal.is_trace`, `proposal.merge_rows`), the gradient of the
  training objective (`proposal.mlp_grad`) and a round's Adam steps
  (`proposal.adam_run`).

The networks are this repository's own generators (cusmc_b200/netgen.py) at
the sizes its benchmark and tests use, and sizes between them.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from cusmc_b200 import api, netgen
from cusmc_b200 import proposal as P


def listed():
    return [
        # a quick look at a small model from a host program: the smallest call
        {"name": "host_random8_100", "kind": "host", "net": "random", "size": 8, "net_seed": 0, "horizon": 100,
         "runs": 100, "query": "prob"},
        # the benchmark's small random network at its own run count
        {"name": "host_random8_10k", "kind": "host", "net": "random", "size": 8, "net_seed": 0, "horizon": 100,
         "runs": 10_000, "query": "prob"},
        # an odd-sized epidemic, a location query, an odd number of runs: a
        # first estimate to a few percent
        {"name": "run_epidemic37_loc_1501", "kind": "run", "net": "epidemic", "size": 37, "net_seed": 0,
         "horizon": 100, "runs": 1501, "query": "loc"},
        # the command line's default number of simulations, expected maximum
        # of the infected on the 100-agent epidemic
        {"name": "run_epidemic100_16k", "kind": "run", "net": "epidemic", "size": 100, "net_seed": 0, "horizon": 100,
         "runs": 16_384, "query": "emax"},
        # the benchmark's headline: a million runs of the 100-agent epidemic
        {"name": "run_epidemic100_1m", "kind": "run", "net": "epidemic", "size": 100, "net_seed": 0, "horizon": 100,
         "runs": 1_000_000, "query": "prob"},
        # timed mutual exclusion (clocks, invariants, guards): mid-sized
        {"name": "run_mutex32_50k", "kind": "run", "net": "mutex", "size": 32, "net_seed": 0, "horizon": 200,
         "runs": 50_000, "query": "prob"},
        # ... and the largest of its sizes
        {"name": "run_mutex256_2k", "kind": "run", "net": "mutex", "size": 256, "net_seed": 0, "horizon": 200,
         "runs": 2000, "query": "prob"},
        # a benchmark suite of uneven random models in one launch
        {"name": "batch_16", "kind": "batch", "net": "random", "size": 16, "net_seed": 1000, "horizon": 0,
         "runs": 16_000, "query": "prob"},
        # weighted runs of a rare event under a proposal: an estimate's bulk
        {"name": "is_run_epidemic100_100k", "kind": "is_run", "net": "epidemic", "size": 100, "net_seed": 0,
         "horizon": 75, "runs": 100_000, "query": "rare"},
        # ... and a training round's runs
        {"name": "is_run_epidemic100_4k", "kind": "is_run", "net": "epidemic", "size": 100, "net_seed": 0,
         "horizon": 75, "runs": 4000, "query": "rare"},
        # the replay of a training round's elite runs into training rows
        {"name": "is_trace_epidemic100_200", "kind": "is_trace", "net": "epidemic", "size": 100, "net_seed": 0,
         "horizon": 75, "runs": 200, "query": "rare"},
        # a training round's Adam steps over its merged rows
        {"name": "adam_150k_rows", "kind": "adam", "net": "", "size": 40, "net_seed": 0, "horizon": 0,
         "runs": 150_001, "query": ""},
    ]


# component-steps of a drawn case by network, so that none costs more than
# the largest listed one
_DRAW_WORK = {"epidemic": 1.0e11, "mutex": 1.5e10, "random": 5.0e9}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "run", "run", "run", "batch", "is_run", "is_run", "is_trace", "adam", "mlp_grad"])
    if kind in ("adam", "mlp_grad"):
        return {"kind": kind, "net": "", "size": rng.randint(5, 40), "net_seed": 0, "horizon": 0,
                "runs": _log_int(rng, 1000, 400_000 if kind == "adam" else 2_000_000), "query": ""}
    if kind == "batch":
        jobs = rng.randint(2, 32)
        return {"kind": kind, "net": "random", "size": jobs, "net_seed": rng.randint(1000, 1031), "horizon": 0,
                "runs": jobs * _log_int(rng, 100, 1000), "query": "prob"}
    if kind in ("is_run", "is_trace"):
        return {"kind": kind, "net": "epidemic", "size": rng.randint(20, 100), "net_seed": 0,
                "horizon": rng.randint(40, 90),
                "runs": _log_int(rng, 500, 100_000) if kind == "is_run" else _log_int(rng, 20, 1000),
                "query": "rare"}
    case = {"kind": kind, "net": rng.choice(["epidemic", "mutex", "random"]), "net_seed": rng.randint(0, 99)}
    case["size"] = {"epidemic": _log_int(rng, 4, 200), "mutex": _log_int(rng, 2, 256),
                    "random": _log_int(rng, 2, 64)}[case["net"]]
    case["horizon"] = rng.randint(50, 200)
    case["runs"] = 1
    most = min(1e6, _DRAW_WORK[case["net"]] / (_steps(case) * case["size"]))
    case["runs"] = _log_int(rng, 64, max(most, 128))
    case["query"] = rng.choice(["prob", "prob", "emax", "loc"] if case["net"] == "epidemic" else ["prob", "emax"])
    return case


def _workload(case):
    if case["net"] == "epidemic":
        return netgen.epidemic(n_agents=case["size"], horizon=case["horizon"], runs=case["runs"],
                               r_threshold=max(1, case["size"] // 2))
    if case["net"] == "mutex":
        return netgen.mutex(case["size"], horizon=case["horizon"], runs=case["runs"])
    return netgen.random_network(case["net_seed"], n_comps=case["size"], horizon=case["horizon"], runs=case["runs"])


def _blob(w, loc_query=""):
    fd, path = tempfile.mkstemp(suffix=".xml")
    os.close(fd)
    try:
        return api.compile_model(w.write(path), loc_query, bool(loc_query))
    finally:
        os.unlink(path)


def _proposal(seed, size):
    """A proposal of the trained network's shape: random hidden layers, a
    mild tilt towards faster rates that depends on the state."""
    prop = P.Proposal.init(seed)
    prop.w3 = (np.random.default_rng(seed + 1).standard_normal(P.HID) * 0.03).astype(np.float32)
    prop.b3 = 0.3
    return prop


def _rows(seed, n, inputs):
    """Training rows as a replay makes them: location class, S/E/I/R
    fractions of `inputs` agents, time in 64 steps of the horizon; a and b
    the weighted rate and winner terms."""
    rng = np.random.default_rng(seed)
    x = np.zeros((n, P.IN), np.float32)
    x[np.arange(n), rng.integers(0, 4, n)] = 1.0
    counts = rng.dirichlet([4, 1, 1, 4], n) * inputs
    x[:, 5:9] = np.floor(counts).astype(np.float32) / np.float32(inputs)
    x[:, 9] = np.floor(rng.uniform(0, 64, n)).astype(np.float32) / np.float32(64)
    rows = np.zeros(n, dtype=np.dtype([("x", "<u2", (P.IN,)), ("a", "<f4"), ("b", "<f4")]))
    rows["x"] = P.f32_to_bf16_bits(x.ravel()).reshape(n, P.IN)
    rows["a"] = rng.exponential(1e-3, n).astype(np.float32)
    rows["b"] = (rng.uniform(0, 1, n) < 0.25).astype(np.float32) * np.float32(1e-3)
    return rows


def prepare(case, seed):
    kind, n = case["kind"], case["runs"]
    st = {"kind": kind, "case": case, "seed": 1 + seed}
    dev = torch.device("cuda")
    if kind in ("adam", "mlp_grad"):
        st["rows"] = torch.from_numpy(_rows(seed, n, case["size"]).view(np.uint8).copy()).to(dev)
        prop = _proposal(seed, case["size"])
        st["params"] = prop.pack()
        st["x0"] = prop.vector()
        st["steps"] = case["size"]
        return st
    if kind == "batch":
        jobs = []
        for i, w in enumerate(netgen.batch_networks(case["size"], base_seed=case["net_seed"])):
            q = api.variable_query(w.var_id, 50, threshold=w.threshold, is_max=True, max_steps=1_000_000)
            jobs.append((api.Network(_blob(w)), q, 1 + seed + i, max(10, n // case["size"])))
        st["batch"] = api.Batch(jobs)
        return st
    w = _workload(case)
    if case["query"] == "loc":
        blob = _blob(w, f"Agent{case['size'] // 2}.R")
        st["query"] = api.location_query(w.horizon)
    else:
        blob = _blob(w)
        if case["query"] == "emax":
            # expected maximum of the infected, of the automata in the
            # critical section or of the first counter
            var = {"epidemic": 2, "mutex": 1, "random": 0}[case["net"]]
            st["query"] = api.variable_query(var, w.horizon, is_max=True, is_estimate=True, max_steps=1_000_000)
        elif case["query"] == "rare":
            st["query"] = api.variable_query(w.var_id, w.horizon, threshold=int(0.94 * case["size"]), is_max=True)
        else:
            st["query"] = api.variable_query(w.var_id, w.horizon, threshold=w.threshold, is_max=True,
                                             max_steps=1_000_000)
    if kind == "host":
        st["blob"] = blob
        return st
    st["net"] = api.Network(blob)
    if kind == "run":
        st["flags"] = torch.empty(n, dtype=torch.uint8, device=dev)
        st["values"] = torch.empty(n, dtype=torch.float64, device=dev)
        return st
    st["params"] = _proposal(seed, case["size"]).pack()
    if kind == "is_trace":
        # a training round's runs, and its elite (about `runs` of them)
        m = 10 * n
        logw = torch.empty(m, dtype=torch.float64, device=dev)
        values = torch.empty(m, dtype=torch.float64, device=dev)
        steps = torch.empty(m, dtype=torch.int32, device=dev)
        P.is_run(st["net"], st["query"], st["params"], st["seed"], m, logw=logw, values=values, steps=steps)
        # (a buffer of twice the expected rows, as long-lived as the loop)
        cap = int(8 * n * _steps(case))
        sel = P.select_elite(values.cpu().numpy(), logw.cpu().numpy(), steps.cpu().numpy().view(np.uint32),
                             st["query"].threshold, max_rows=cap)
        st["runs"] = torch.from_numpy(sel.runs.copy()).to(dev)
        st["weights"] = torch.from_numpy(sel.weights).to(dev)
        st["offset"] = torch.from_numpy(sel.row_offset.view(np.int64)).to(dev)
        st["n_rows"] = sel.n_rows
        st["rows"] = torch.zeros(cap * P.ROW_BYTES, dtype=torch.uint8, device=dev)
        st["merged"] = torch.zeros_like(st["rows"])
        return st
    st["flags"] = torch.empty(n, dtype=torch.uint8, device=dev)
    st["logw"] = torch.empty(n, dtype=torch.float64, device=dev)
    st["values"] = torch.empty(n, dtype=torch.float64, device=dev)
    st["steps"] = torch.empty(n, dtype=torch.int32, device=dev)
    return st


def _result(r):
    return {"hits": int(r.hits), "steps": int(r.steps), "capped": int(r.capped), "sum": float(r.sum),
            "sum_sq": float(r.sum_sq), "estimate": float(r.estimate)}


def run(st):
    kind, n = st["kind"], st["case"]["runs"]
    if kind == "host":
        r, flags, values, _ = api.run_host(st["blob"], st["query"], st["seed"], n)
        return {"flags": flags, "values": values, **_result(r)}
    if kind == "run":
        r = st["net"].run(st["query"], st["seed"], n, flags=st["flags"], values=st["values"])
        return {"flags": st["flags"], "values": st["values"], **_result(r)}
    if kind == "batch":
        res = st["batch"].run()
        outs = [st["batch"].outputs(i) for i in range(len(res))]
        out = {k: np.concatenate([o[k] for o in outs]) for k in ("flags", "values", "steps")}
        totals = [_result(r) for r in res]
        return {**out, **{"job_" + k: np.array([t[k] for t in totals]) for k in totals[0]}}
    if kind == "is_run":
        r = P.is_run(st["net"], st["query"], st["params"], st["seed"], n, flags=st["flags"], logw=st["logw"],
                     values=st["values"], steps=st["steps"])
        return {"flags": st["flags"], "logw": st["logw"], "values": st["values"], "run_steps": st["steps"],
                **_result(r)}
    if kind == "is_trace":
        P.is_trace(st["net"], st["query"], st["params"], st["seed"], st["runs"], st["weights"], st["offset"],
                   st["rows"])
        m = P.merge_rows(st["rows"], st["offset"], len(st["runs"]), st["n_rows"], st["merged"])
        return {"rows": st["rows"], "merged_rows": m, "merged": st["merged"]}
    if kind == "adam":
        x, opt = st["x0"].copy(), P.AdamState()
        j0, j1 = P.adam_run(st["rows"], n, st["steps"], 3e-2, x, opt)
        return {"x": x, "m": opt.m, "v": opt.v, "j_first": j0, "j_last": j1}
    g, j = P.mlp_grad(st["params"], st["rows"], n)
    return {"grad": g, "objective": j}


def _steps(case):
    """Race steps of one run, from the networks' rates (a delay of rate r
    comes every 1 / (r ln 2) of model time)."""
    n, T, ln2 = case["size"], case["horizon"], math.log(2.0)
    if case["net"] == "epidemic":
        # mean-field S, E, I, R in unit time steps; R agents tick with rate 1
        s, e, i, r, steps = n - 1.0, 0.0, 1.0, 0.0, 0.0
        for _ in range(int(T)):
            a, b, c = ln2 * 0.3 * s * i / n, ln2 * 0.2 * e, ln2 * 0.1 * i
            steps += a + b + c + ln2 * r
            s, e, i, r = s - a, e + a - b, i + b - c, r + c
        return max(steps, 1.0)
    return max(ln2 * T * n * (1.0 if case["net"] == "mutex" else 0.3), 1.0)


# integer and floating-point operations of one component's part in a race:
# its share of a ten-round Philox4x32 block (four products and four
# exclusive-ors a round, for four components) and one comparison
_COMPONENT_OPS = 10 * 8 / 4 + 1
# multiply-adds of the proposal network for one row, forward, and with the
# gradient (back-propagation and the weights' outer products)
_MLP_FORWARD = 16 * 64 + 64 * 64 + 64
_MLP_GRAD = 2 * _MLP_FORWARD + 64 * 64


def work(case):
    kind, n = case["kind"], case["runs"]
    if kind in ("adam", "mlp_grad"):
        passes = case["size"] if kind == "adam" else 1
        return {"bytes": P.ROW_BYTES * n + 5 * 4 * P.GRAD_FLOATS, "flops": 2 * _MLP_GRAD * n * passes}
    if kind == "batch":
        ops = 0.0
        for w in netgen.batch_networks(case["size"], base_seed=case["net_seed"]):
            comps = w.n_vars - 2
            one = {"net": "random", "size": comps, "horizon": 50}
            ops += _steps(one) * comps * _COMPONENT_OPS * max(10, n // case["size"])
        return {"bytes": 13 * n + 100_000, "flops": ops}
    ops = n * _steps(case) * case["size"] * _COMPONENT_OPS
    per_run = {"host": 9, "run": 9, "is_run": 21, "is_trace": 4 * P.ROW_BYTES * _steps(case)}[kind]
    return {"bytes": per_run * n + 230 * case["size"], "flops": ops}


def _exact_grad(rows, prop):
    """J and its gradient in 64 bits (BF16 weights as the network has them)."""
    d = torch.float64
    w1 = torch.from_numpy(P.bf16_bits_to_f32(P.f32_to_bf16_bits(prop.w1))).to(d)
    w2 = torch.from_numpy(P.bf16_bits_to_f32(P.f32_to_bf16_bits(prop.w2))).to(d)
    b1, b2, w3 = (torch.from_numpy(v).to(d) for v in (prop.b1, prop.b2, prop.w3))
    g = [torch.zeros_like(v) for v in (w1, b1, w2, b2, w3)]
    g3, objective = 0.0, 0.0
    c, k = math.sqrt(2.0 / math.pi), 0.044715

    def gelu(z):
        s = torch.sigmoid(2 * c * (z + k * z ** 3))
        return z * s, s + z * s * (1 - s) * 2 * c * (1 + 3 * k * z * z)

    for lo in range(0, len(rows), 65536):
        part = rows[lo:lo + 65536]
        x = torch.from_numpy(P.bf16_bits_to_f32(part["x"])).to(d)
        a, b = (torch.from_numpy(part[f].astype(np.float64)) for f in ("a", "b"))
        h1, d1 = gelu(x @ w1.T + b1)
        h2, d2 = gelu(h1 @ w2.T + b2)
        theta = h2 @ w3 + float(np.float32(prop.b3))
        clipped = theta.clamp(-4.0, 4.0)
        e = torch.exp(clipped)
        objective += float((b * clipped - a * e).sum())
        gt = torch.where(theta == clipped, b - a * e, torch.zeros_like(a))
        z2 = gt[:, None] * w3 * d2
        z1 = (z2 @ w2) * d1
        for acc, v in zip(g, (z1.T @ x, z1.sum(0), z2.T @ h1, z2.sum(0), h2.T @ gt)):
            acc += v
        g3 += float(gt.sum())
    return np.concatenate([v.numpy().ravel() for v in g] + [np.array([g3])]), objective


def exact(case, seed):
    """Only the gradient is a number that arithmetic in 64 bits gives: a
    run's flag, value and weight are defined by its random stream and its
    own operations, and a sequence of Adam steps by the gradients before."""
    if case["kind"] != "mlp_grad":
        return None
    grad, objective = _exact_grad(_rows(seed, case["runs"], case["size"]), _proposal(seed, case["size"]))
    return {"grad": grad, "objective": objective}
