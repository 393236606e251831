"""GPU parity of the drop-in search's small form (32-bit labels, all state in
one SM) at its block sizes, at the last graph that fits and the first that
does not, with costs too large for it, and under a bounded number of rounds."""

import numpy as np
import pytest

import apgar_b200
import oracle
from apgar_b200 import dropin
from tests.test_dropin_large_gpu import _board, _queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [8, 16, 17, 32, 33, 58, 59, 60])
@pytest.mark.parametrize("surcharge,rounds", [(0, 100_000), (1 << 33, 100_000), (0, 60_000)])
def test_paths_and_workspaces_match_the_oracle(side, surcharge, rounds):
    header, layers, nodes, runs, run_nodes, cut = _board(side, side, 3)
    view = dropin.View(header, layers, nodes, runs, run_nodes)
    entries = _queries(nodes, cut, side, 6)
    for e in entries[::2]:
        e["diagonal_step_surcharge"] = surcharge
    S = 9 * view.node_count
    for generator in (dropin.GENERATOR_PERSISTENT, dropin.GENERATOR_FRONTIER):
        queries, edges = dropin.make_queries(view.node_count, entries, generator=generator, maximum_rounds=rounds)
        pending = view.execute_batch(queries, edges, generator=generator, maximum_rounds=rounds)
        results, compact, states, _ = pending.readback()
        if generator == dropin.GENERATOR_FRONTIER:
            labels, preds, owners, _ = pending.readback_workspace()
        pending.close()
        for i, e in enumerate(entries):
            args = (e.get("orthogonal_step_surcharge", 0), e.get("diagonal_step_surcharge", 0),
                    e.get("bend_surcharge", 0), e.get("policy"))
            ok, _, goal_state, path, exact = oracle.graph_search(nodes, (10, 14, 3), e["start_node"], e["goal_node"],
                                                                 *args, want_labels=True)
            done = apgar_b200.COMPLETION_REACHED if ok else apgar_b200.COMPLETION_DISCONNECTED
            assert results[i]["completion"] == done, i
            if generator == dropin.GENERATOR_FRONTIER:
                sl = slice(i * S, (i + 1) * S)
                assert np.array_equal(labels[sl], exact), i
                assert np.array_equal(preds[sl], oracle.graph_predecessors(nodes, (10, 14, 3), e["start_node"], exact,
                                                                           *args)), i
                assert (owners[sl] == i + 1).all()
            elif ok:
                c = compact[i]
                assert results[i]["goal_state"] == goal_state
                assert np.array_equal(states[int(c["state_offset"]):][:int(c["state_count"])], path), i
    view.close()


def test_a_budget_of_rounds_ends_the_search():
    header, layers, nodes, runs, run_nodes, cut = _board(36, 5, 0)
    view = dropin.View(header, layers, nodes, runs, run_nodes)
    entries = _queries(nodes, cut, 9, 6)
    queries, edges = dropin.make_queries(view.node_count, entries, generator=dropin.GENERATOR_PERSISTENT,
                                         maximum_rounds=2)
    pending = view.execute_batch(queries, edges, generator=dropin.GENERATOR_PERSISTENT, maximum_rounds=2)
    results, compact, _, _ = pending.readback()
    pending.close()
    view.close()
    assert (results["rounds"] == 2).all()
    assert (results["completion"] == apgar_b200.COMPLETION_BUDGET_EXHAUSTED).all()
    assert (compact["state_count"] == 0).all()
