"""Broadcasts in lane groups: a step keeps its receivers' edge sets where the
components' delay records lie, and the winner's lane has written its record
just before.  Networks in which most transitions broadcast, every other
component receives and every record changes with the rate table, in each share
of a full warp, in two narrower groups and in a batch: the traces equal the
CPU oracle's bit for bit."""
import os
import tempfile

import numpy as np
import pytest

import oracle
from cusmc_b200 import api, netgen

pytestmark = pytest.mark.gpu


def _blob(n_comps):
    d = netgen._Doc("int v0 = 1;\nbroadcast chan bc;")
    for c in range(n_comps):
        a, b = d.new_id(), d.new_id()
        # a sends, b falls back when it hears a sender and on its own
        rate = "0.02 * v0" if c % 3 else f"0.{1 + c % 7}"
        d.template(f"C{c}", "clock x;",
                   [(a, "A", [("exponentialrate", rate)]), (b, "B", [("exponentialrate", "0.3")])], a if c % 2 else b,
                   [(a, b, [("synchronisation", "bc!"), ("assignment", "v0 = v0 + 1, x = 0")]),
                    (b, a, [("guard", "x >= 0"), ("synchronisation", "bc?")]),
                    (b, a, [("assignment", "v0 = 1, x = 0")])])
    with tempfile.NamedTemporaryFile("w", suffix=".xml", delete=False) as f:
        f.write(d.finish())
    try:
        return api.compile_model(f.name)
    finally:
        os.unlink(f.name)


QUERY = dict(threshold=3, is_max=True, max_steps=400)


@pytest.mark.parametrize("n_comps,g,k", [(29, 32, 1), (61, 32, 2), (127, 32, 4), (200, 32, 8), (300, 32, 16),
                                         (13, 16, 1), (63, 16, 4)])
def test_broadcasts_in_lane_groups_give_the_oracle_traces(n_comps, g, k):
    blob = _blob(n_comps)
    q = api.variable_query(0, 20, **QUERY)
    _, want, _ = oracle.run(blob, q, 3, 300, threads=0, digests=True, final_state=True)
    net = api.Network(blob)
    try:
        net.set_plan(0, g, k, 128)
        r, got = net.run_verify(q, 3, 300)
        assert (r.family, r.lanes_per_run, r.comps_per_lane) == (0, g, k)
    finally:
        net.close()
    for key in ("steps", "flags", "digests", "final_state"):
        assert np.array_equal(got[key], want[key]), key


def test_broadcasts_in_batches_give_the_oracle_traces():
    q = api.variable_query(0, 20, **QUERY)
    blobs = [_blob(n) for n in (29, 127, 200)]
    nets = [api.Network(b) for b in blobs]
    batch = api.Batch([(n, q, 5 + i, 200) for i, n in enumerate(nets)], verify=True)
    try:
        batch.set_group_comps(2)
        batch.run()
        outs = [batch.outputs(i) for i in range(3)]
    finally:
        batch.close()
        for n in nets:
            n.close()
    for i, blob in enumerate(blobs):
        _, want, _ = oracle.run(blob, q, 5 + i, 200, threads=0, digests=True, final_state=True)
        for key in ("steps", "flags", "digests"):
            assert np.array_equal(outs[i][key], want[key]), (i, key)
        assert np.array_equal(outs[i]["final_state"].ravel(), np.asarray(want["final_state"]).ravel())
