"""GPU parity of the frontier's tile form (32 x 32 units) where it can go
wrong: windows at the edges of a unit, mazes that take many sweeps, move costs
on both sides of a straight move, and its slot workspace with idle warps
visiting other nets.  Costs and canonical paths are integers and must equal
the oracle's exactly."""

import numpy as np
import pytest

import apgar_b200
import oracle
from apgar_b200 import synth

pytestmark = pytest.mark.gpu


def _check(lat, nets):
    dev = apgar_b200.DeviceLattice(lat)
    try:
        plan = dev.plan(nets, generator="frontier")
        cost_o, paths_o = oracle.dijkstra_batch(lat, nets)
        for _ in range(2):  # the second execution finds the first one's labels
            plan.execute()
            res, paths = plan.readback()
            assert np.array_equal(res["cost"], cost_o), np.flatnonzero(res["cost"] != cost_o)[:10]
            per = apgar_b200.split_paths(res, paths)
            for i in range(len(nets)):
                if cost_o[i] != oracle.lo_inf():
                    assert np.array_equal(per[i], paths_o[i]), i
        plan.close()
    finally:
        dev.close()


def _windows(lat, w, h, count, seed):
    """Nets between free cells of w x h windows placed at random."""
    rng = np.random.default_rng(seed)
    free = ~lat.blocked_dense()
    nets = np.zeros(count, synth.NET_DTYPE)
    for n in nets:
        ls = ()
        while len(ls) == 0:  # a window with a free cell
            x0, y0 = int(rng.integers(0, lat.width - w + 1)), int(rng.integers(0, lat.height - h + 1))
            ls, ys, xs = np.nonzero(free[:, y0:y0 + h, x0:x0 + w])
        a, b = rng.integers(0, len(ls), size=2)
        n["start_layer"], n["start_x"], n["start_y"] = ls[a], x0 + xs[a], y0 + ys[a]
        n["goal_layer"], n["goal_x"], n["goal_y"] = ls[b], x0 + xs[b], y0 + ys[b]
        n["win_x0"], n["win_y0"], n["win_w"], n["win_h"] = x0, y0, w, h
    return nets


@pytest.mark.parametrize("layers", [1, 3, 8])
@pytest.mark.parametrize("w,h", [(1, 1), (1, 65), (31, 33), (32, 32), (33, 31), (64, 96), (65, 97), (128, 1)])
def test_windows_at_the_edges_of_a_unit(layers, w, h):
    lat = synth.make_lattice(100 + layers, layers, 160, 0.2, via_mask=layers > 1)
    _check(lat, _windows(lat, w, h, 12, w * 131 + h))


@pytest.mark.parametrize("orth,diag,via", [(10, 14, 50), (10, 25, 7), (10, 6, 3), (7, 7, 1), (1, 2, 200), (400, 100, 9)])
def test_move_costs_on_both_sides_of_a_straight_move(orth, diag, via):
    base = synth.make_lattice(7, 3, 128, 0.25, via_mask=True)
    lat = synth.Lattice(3, 128, 128, base.blocked, base.via_ok, orth, diag, via)
    _check(lat, synth.make_nets(lat, 8, 40, hpwl_median=60.0, hpwl_sigma=0.6, margin=20))


@pytest.mark.parametrize("layers", [1, 2])
def test_mazes_take_many_sweeps(layers):
    # serpentines of one-cell corridors: every unit is swept many times
    size = 96
    dense = np.zeros((layers, size, size), bool)
    dense[0, 1::2] = True
    dense[0, 1::4, size - 1] = False
    dense[0, 3::4, 0] = False
    if layers == 2:
        dense[1, :, 1::2] = True
        dense[1, size - 1, 1::4] = False
        dense[1, 0, 3::4] = False
    via_ok = None
    if layers == 2:
        allowed = np.zeros((1, size, size), bool)
        allowed[0, ::32, ::32] = True
        via_ok = synth.pack_bits(allowed)
    lat = synth.Lattice(layers, size, size, synth.pack_bits(dense), via_ok)
    # one long path at a time: the batch's path arena holds 8 (w + h) + 64 L cells a net
    short = [(0, x, 0, layers - 1, x, 0, 0, 0, size, size) for x in (0, 2)]
    for long in ((0, 0, 0, 0, 0, 94, 0, 0, size, size), (0, 95, 94, 0, 3, 2, 0, 0, size, size)):
        _check(lat, np.array([long, *short], dtype=synth.NET_DTYPE))


def test_few_slots_and_many_guests(monkeypatch):
    # slots for a handful of nets: every other warp only visits
    lat = synth.make_lattice(61, 3, 512, 0.22, via_mask=True)
    nets = synth.make_nets(lat, 62, 60, hpwl_median=150.0, hpwl_sigma=0.7)
    monkeypatch.setenv("APGAR_B200_FRONTIER_PER_NET_BYTES", "1")
    monkeypatch.setenv("APGAR_B200_FRONTIER_SLOT_BYTES", str(24 << 20))
    _check(lat, nets)


CELL_FORM = (1 << 30) - 1  # a bound on the rounds: the search over single cells


@pytest.mark.parametrize("high", [0, (1 << 29) - 1, 1 << 29, (1 << 31) - 1])
@pytest.mark.parametrize("layers,width,height", [(1, 96, 65), (3, 160, 130)])
def test_priced_results_equal_the_cell_forms(layers, width, height, high):
    # sparse congestion prices, and a few cells priced around the limit at
    # which the tile form hands a net over to the cell form
    import torch

    base = synth.make_lattice(300 + layers, layers, 160, 0.2, via_mask=layers > 1)
    lat = synth.Lattice(layers, height, width, np.ascontiguousarray(base.blocked[:, :height, :width // 32]),
                        None if layers == 1 else np.ascontiguousarray(base.via_ok[:, :height, :width // 32]))
    nets = synth.make_nets(lat, 301, 48, hpwl_median=50.0, hpwl_sigma=0.6, margin=12)
    rng = np.random.default_rng(302)
    cells = layers * height * width
    price = np.where(rng.random(cells) < 0.2, rng.integers(1, 900, cells), 0).astype(np.uint32)
    if high:
        price[rng.integers(0, cells, size=8)] = high
    prices = torch.from_numpy(price.view(np.int32)).cuda()
    dev = apgar_b200.DeviceLattice(lat)
    try:
        out = []
        for rounds in (1 << 30, CELL_FORM):
            plan = dev.plan(nets, generator="frontier", max_rounds=rounds)
            for costs in (prices, None, prices):  # prices come, go and come back
                plan.set_cell_costs(costs)
                plan.execute()
                res, paths = plan.readback()
                out.append((res, paths.copy()))
            plan.close()
    finally:
        dev.close()
    for (a, pa), (b, pb) in zip(out[:3], out[3:]):
        for field in ("cost", "completion", "path_len", "path_offset"):
            assert np.array_equal(a[field], b[field]), field
        assert np.array_equal(pa, pb)


@pytest.mark.parametrize("layers,size,hpwl,margin", [(1, 2112, 1500, 400), (2, 640, 300, 90), (3, 160, 40, 9)])
@pytest.mark.parametrize("priced", [False, True])
def test_corridor_outcomes_equal_the_cell_forms(layers, size, hpwl, margin, priced):
    # coarse cells from 4 to 64 lattice cells a side (a unit holds 64 to part of one)
    import torch

    from apgar_b200 import corridor

    lat = synth.make_lattice(400 + layers, layers, size, 0.2, via_mask=layers > 1)
    nets = synth.make_nets(lat, 401, 24, hpwl_median=float(hpwl), hpwl_sigma=0.3, margin=margin)
    if size == 2112:
        assert max(corridor.coarse_shift(int(n["win_w"]), int(n["win_h"])) for n in nets) >= 5
    rng = np.random.default_rng(402)
    masks = np.concatenate([corridor.segment_corridor(nets[:8], 0), corridor.segment_corridor(nets[8:16], 2),
                            corridor.segment_corridor(nets[16:], 5)])
    masks &= rng.random(masks.shape) < 0.97
    bits = torch.from_numpy(corridor.pack(masks).view(np.int32)).cuda().view(torch.uint32)
    prices = None
    if priced:
        cells = layers * size * size
        price = np.where(rng.random(cells) < 0.1, rng.integers(1, 60, cells), 0).astype(np.uint32)
        prices = torch.from_numpy(price.view(np.int32)).cuda()
    dev = apgar_b200.DeviceLattice(lat)
    try:
        out = []
        for rounds in (1 << 30, CELL_FORM):
            plan = dev.plan(nets, generator="frontier", max_rounds=rounds)
            plan.set_cell_costs(prices)
            plan.set_corridors(bits)
            plan.execute()
            res, paths = plan.readback()
            out.append((res, paths.copy(), plan.corridor_status()))
            plan.close()
    finally:
        dev.close()
    (a, pa, sa), (b, pb, sb) = out
    assert np.array_equal(sa, sb), (sa, sb)
    assert len(set(sa.tolist())) > 1
    for field in ("cost", "completion", "path_len"):
        assert np.array_equal(a[field], b[field]), field
    assert np.array_equal(pa, pb)
