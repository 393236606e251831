"""Cancellation of a running batch in each form of the search: every net that
comes back is cancelled or exact, a large batch does not run to its end, and
the next call is exact."""

import numpy as np
import pytest

import apgar_b200
import oracle
from apgar_b200 import dropin, synth
from tests.test_dropin_large_gpu import _board, _queries

pytestmark = pytest.mark.gpu

SLOTS = {"APGAR_B200_FRONTIER_PER_NET_BYTES": "1", "APGAR_B200_FRONTIER_SLOT_BYTES": str(256 << 20)}
CELL_FORM = (1 << 30) - 1  # a bound on the rounds: the search over single cells


@pytest.mark.parametrize("form", ["tiles", "teams", "slots", "cells", "sweep"])
def test_a_cancelled_batch_is_cancelled_or_exact(monkeypatch, form):
    lat = synth.make_lattice(91, 4, 1024, 0.25, pads=True)
    nets = synth.make_nets(lat, 92, 2000, hpwl_median=250.0, hpwl_sigma=0.6)
    options = {"tiles": dict(generator="frontier"), "slots": dict(generator="frontier"),
               "teams": dict(generator="frontier", class_bounds=apgar_b200.class_bounds(6, 8, 10, 12)),
               "cells": dict(generator="frontier", max_rounds=CELL_FORM), "sweep": dict()}[form]
    if form == "slots":
        for name, value in SLOTS.items():
            monkeypatch.setenv(name, value)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        exact, paths = dev.route(nets, **options)
        exact_paths = apgar_b200.split_paths(exact, paths)
        assert not (exact["completion"] == apgar_b200.COMPLETION_CANCELLED).any()
        res, paths = dev.route(nets, cancel=np.ones(1, np.uint32), **options)
        cancelled = res["completion"] == apgar_b200.COMPLETION_CANCELLED
        assert cancelled.any()
        for i, path in enumerate(apgar_b200.split_paths(res, paths)):
            if cancelled[i]:
                assert path is None and res[i]["cost"] == oracle.lo_inf()
            else:
                assert res[i]["cost"] == exact[i]["cost"] and res[i]["completion"] == exact[i]["completion"]
                assert (path is None) == (exact_paths[i] is None)
                assert path is None or np.array_equal(path, exact_paths[i])
        again, paths = dev.route(nets, **options)
        for field in ("cost", "completion", "path_len", "path_offset"):
            assert np.array_equal(again[field], exact[field]), field
        assert all((a is None) == (b is None) and (a is None or np.array_equal(a, b))
                   for a, b in zip(apgar_b200.split_paths(again, paths), exact_paths))
    finally:
        dev.close()


@pytest.mark.parametrize("side", [40, 62])  # the small form and the one in global memory
@pytest.mark.parametrize("generator", [dropin.GENERATOR_PERSISTENT, dropin.GENERATOR_FRONTIER])
def test_a_cancelled_candidate_batch_is_cancelled_or_exact(side, generator):
    header, layers, nodes, runs, run_nodes, cut = _board(side, side, 3)
    view = dropin.View(header, layers, nodes, runs, run_nodes)
    queries, edges = dropin.make_queries(view.node_count, _queries(nodes, cut, side, 400), generator=generator)
    out = []
    for cancel in (None, np.ones(1, np.uint8), None):
        pending = view.execute_batch(queries, edges, generator=generator, cancel=cancel)
        results, compact, states, _ = pending.readback()
        pending.close()
        out.append((results, compact, states))
    view.close()
    exact, (res, compact, states), again = out
    cancelled = res["completion"] == apgar_b200.COMPLETION_CANCELLED
    assert not (exact[0]["completion"] == apgar_b200.COMPLETION_CANCELLED).any()
    assert cancelled.any()
    for i in np.flatnonzero(~cancelled):
        assert res[i]["completion"] == exact[0][i]["completion"] and res[i]["goal_state"] == exact[0][i]["goal_state"]
        a, b = compact[i], exact[1][i]
        assert np.array_equal(states[int(a["state_offset"]):][:int(a["state_count"])],
                              exact[2][int(b["state_offset"]):][:int(b["state_count"])])
    for field in ("completion", "goal_state"):
        assert np.array_equal(again[0][field], exact[0][field]), field
    assert np.array_equal(again[2], exact[2])
