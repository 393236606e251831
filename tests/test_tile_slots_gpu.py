"""The tile search's slot workspace: no more slots than nets, and the same
routes as with a workspace per net for prices, own-route pricing and kept
routes.  Results are integers and must be equal exactly."""

import numpy as np
import pytest

import apgar_b200
from apgar_b200 import negotiate, prices, synth

pytestmark = pytest.mark.gpu


def _words(lat, net):
    """32-bit words of a net's tile workspace: labels, four words a unit, the queue's ring."""
    units = lat.layers * -(-int(net["win_w"]) // 32) * -(-int(net["win_h"]) // 32)
    ring = 32
    while ring < units:
        ring *= 2
    return (units * 1028 + ring + 31) & ~31


@pytest.mark.parametrize("count", [1, 5, 60])
def test_no_more_slots_than_nets(monkeypatch, count):
    lat = synth.make_lattice(71, 3, 512, 0.2, via_mask=True)
    nets = synth.make_nets(lat, 72, count, hpwl_median=150.0, hpwl_sigma=0.7)
    monkeypatch.setenv("APGAR_B200_FRONTIER_PER_NET_BYTES", "1")
    dev = apgar_b200.DeviceLattice(lat)
    try:
        plan = dev.plan(nets, generator="frontier")
        assert plan.info()["label_cells"] <= count * max(_words(lat, n) for n in nets)
        plan.execute()
        slots = plan.readback()
        plan.close()
        monkeypatch.delenv("APGAR_B200_FRONTIER_PER_NET_BYTES")
        plan = dev.plan(nets, generator="frontier")
        plan.execute()
        own = plan.readback()
        plan.close()
        for field in ("cost", "completion", "path_len"):
            assert np.array_equal(slots[0][field], own[0][field]), field
        assert np.array_equal(slots[1], own[1])
    finally:
        dev.close()


@pytest.mark.parametrize("partial", [False, True])
def test_negotiated_rounds_in_slots(monkeypatch, partial):
    lat = synth.make_lattice(81, 4, 384, 0.22, pads=True)
    segments, _ = synth.make_multi_terminal_nets(lat, 82, 120, 90.0, 0.8)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        out = []
        for env in ({}, {"APGAR_B200_FRONTIER_PER_NET_BYTES": "1"},
                    {"APGAR_B200_FRONTIER_PER_NET_BYTES": "1", "APGAR_B200_FRONTIER_SLOT_BYTES": str(16 << 20)}):
            with monkeypatch.context() as m:
                for name, value in env.items():
                    m.setenv(name, value)
                plan = dev.plan(segments, generator="frontier")
            n = negotiate.Negotiation(plan, prices.policy(capacity=1))
            n.run(5, partial=partial)
            usage, history, costs, _ = n.readback()
            res, paths = plan.readback()
            out.append((plan.info()["label_cells"], res["cost"], res["completion"], paths, usage, history, costs))
            n.close()
            plan.close()
        assert len({o[0] for o in out}) == 3  # three different workspaces
        for o in out[1:]:
            assert all(np.array_equal(a, b) for a, b in zip(out[0][1:], o[1:]))
    finally:
        dev.close()
