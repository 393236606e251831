"""Prices come to and go from a resident frontier plan at any time: the plan
keeps its form and its buffers, so setting them allocates nothing, is allowed
while a stream is captured, and leaves graphs captured from the plan valid.
Nets that the tile search hands over are decided with their own class's level
width.  Results are integers and must be equal exactly."""

import numpy as np
import pytest

import apgar_b200
import oracle
from apgar_b200 import autotune, negotiate, prices, synth

pytestmark = pytest.mark.gpu

CELL_FORM = (1 << 30) - 1  # a bound on the rounds: the search over single cells
# windows above 2^12 cells are a whole CTA's; their levels are as wide as the others', or wider
BOUNDS = apgar_b200.class_bounds(6, 8, 10, 12)
SCHEDULES = [autotune.Schedule(class_bounds=BOUNDS), autotune.Schedule(class_bounds=BOUNDS, wide_bucket_width=400)]


def _board(seed):
    lat = synth.make_lattice(seed, 3, 160, 0.2, via_mask=True)
    nets = synth.make_nets(lat, seed + 1, 48, hpwl_median=50.0, hpwl_sigma=0.6, margin=12)
    cells = 3 * nets["win_w"].astype(int) * nets["win_h"]
    assert 0 < (cells > 1 << 12).sum() < len(nets)  # both kinds of nets
    return lat, nets


def _prices(lat, seed, high=0):
    import torch

    rng = np.random.default_rng(seed)
    cells = lat.layers * lat.height * lat.width
    price = np.where(rng.random(cells) < 0.2, rng.integers(1, 900, cells), 0).astype(np.uint32)
    if high:
        price[rng.integers(0, cells, size=30)] = high
    return torch.from_numpy(price.view(np.int32)).cuda()


def _results(plan):
    res, paths = plan.readback()
    return [res[k].copy() for k in ("cost", "completion", "path_len", "path_offset")] + [paths.copy()]


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("schedule", SCHEDULES)
def test_prices_allocate_nothing(schedule):
    import torch

    lat, nets = _board(500)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        plan = dev.plan(nets, generator="frontier", schedule=schedule)
        costs = _prices(lat, 501)
        torch.cuda.synchronize()
        before, free = plan.info(), torch.cuda.mem_get_info()[0]
        plan.set_cell_costs(costs)
        assert plan.info() == before and torch.cuda.mem_get_info()[0] == free
        n = negotiate.Negotiation(plan, prices.policy(capacity=1))
        assert plan.info() == before
        n.close()
        plan.close()
    finally:
        dev.close()


@pytest.mark.parametrize("schedule", SCHEDULES)
def test_prices_are_set_while_a_stream_is_captured(schedule):
    import torch

    lat, nets = _board(510)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        plan = dev.plan(nets, generator="frontier", schedule=schedule)
        costs = _prices(lat, 511)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.set_cell_costs(costs)
            plan.execute(torch.cuda.current_stream().cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        replayed = _results(plan)
        plan.execute()
        assert _equal(replayed, _results(plan))
        plan.set_cell_costs(None)
        plan.execute()
        assert not np.array_equal(replayed[0], _results(plan)[0])
        plan.close()
    finally:
        dev.close()


@pytest.mark.parametrize("schedule", SCHEDULES)
def test_a_captured_execution_outlives_prices(schedule):
    import torch

    lat, nets = _board(520)
    cost_o, _ = oracle.dijkstra_batch(lat, nets)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        plan = dev.plan(nets, generator="frontier", schedule=schedule)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.execute(torch.cuda.current_stream().cuda_stream)
        plan.set_cell_costs(_prices(lat, 521))
        plan.execute()
        plan.readback()
        n = negotiate.Negotiation(plan, prices.policy(capacity=1))
        n.run(3, use_graph=True, partial=True)
        n.readback()
        n.close()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(plan.readback()[0]["cost"], cost_o)
        plan.close()
    finally:
        dev.close()


@pytest.mark.parametrize("high", [0, 1 << 29, (1 << 31) - 1])
@pytest.mark.parametrize("schedule", SCHEDULES)
def test_handed_over_nets_keep_their_level_width(schedule, high):
    lat, nets = _board(530)
    costs = _prices(lat, 531, high)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        out = []
        for rounds in (1 << 30, CELL_FORM):
            plan = dev.plan(nets, generator="frontier", max_rounds=rounds, schedule=schedule)
            plan.set_cell_costs(costs)
            for _ in range(2):
                plan.execute()
                out.append(_results(plan))
            plan.close()
        assert all(_equal(out[0], o) for o in out[1:])
        if high == (1 << 31) - 1:
            assert (out[0][1] == apgar_b200.COMPLETION_REJECTED).any()
    finally:
        dev.close()
