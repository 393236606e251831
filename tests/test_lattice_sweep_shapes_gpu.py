"""Every shape of the sweep kernel (cells per lane, warps side by side, layers)
at the edges of its row widths, in both frames, against the oracle: costs,
canonical paths and the schedule's counters are integers and must be equal."""

import numpy as np
import pytest

import apgar_b200
import oracle
from apgar_b200 import synth

pytestmark = pytest.mark.gpu


def _pack(dense):
    return np.ascontiguousarray(np.packbits(dense, axis=-1, bitorder="little")).view(np.uint32)


def _lattice(layers, height, width, seed, via_mask, costs=(10, 14, 50)):
    rng = np.random.default_rng(seed)
    width = -(-width // 32) * 32
    via = _pack(rng.random((layers - 1, height, width)) < 0.7) if via_mask and layers > 1 else None
    return synth.Lattice(layers, height, width, _pack(rng.random((layers, height, width)) < 0.15), via, *costs)


def _nets(lat, w, h, count, seed):
    rng = np.random.default_rng(seed)
    free = ~lat.blocked_dense()
    nets = np.zeros(count, synth.NET_DTYPE)
    for n in nets:
        x0, y0 = int(rng.integers(0, lat.width - w + 1)), int(rng.integers(0, lat.height - h + 1))
        ls, ys, xs = np.nonzero(free[:, y0:y0 + h, x0:x0 + w])
        a, b = rng.integers(0, max(len(ls), 1), size=2) if len(ls) else (0, 0)
        if len(ls):
            n["start_layer"], n["start_x"], n["start_y"] = ls[a], x0 + xs[a], y0 + ys[a]
            n["goal_layer"], n["goal_x"], n["goal_y"] = ls[b], x0 + xs[b], y0 + ys[b]
        else:  # no free cell: a rejected or disconnected net
            n["start_x"] = n["goal_x"] = x0
            n["start_y"] = n["goal_y"] = y0
        n["win_x0"], n["win_y0"], n["win_w"], n["win_h"] = x0, y0, w, h
    return nets


def _check(lat, nets):
    dev = apgar_b200.DeviceLattice(lat)
    try:
        res, paths = dev.route(nets, generator="sweep")
    finally:
        dev.close()
    paths = apgar_b200.split_paths(res, paths)
    cost_o, paths_o = oracle.dijkstra_batch(lat, nets)
    _, st = oracle.sweep_batch(lat, nets)
    assert np.array_equal(res["cost"], cost_o)
    for i in range(len(nets)):
        if cost_o[i] != oracle.lo_inf():
            assert np.array_equal(paths[i], paths_o[i]), i
    ran = st[:, 0] > 0
    for field, column in (("sweeps", 0), ("row_steps", 1), ("row_stores", 2), ("row_loads", 5)):
        assert np.array_equal(res[field][ran], st[ran, column].astype(np.uint32)), field


WIDEST = {1: 8192, 2: 4096, 3: 2048, 4: 2048, 6: 1024, 8: 1024}


@pytest.mark.parametrize("layers", sorted(WIDEST))
def test_rows_at_the_edges_of_a_shape(layers):
    widths = [1, 3, 4, 127, 128, 129, 255, 257, 511, 512, 513, 767, 769, 1023, 1024, 1025, 1537, 2047, 2049, 2561,
              4095, 5121, 8191, WIDEST[layers]]
    for k, w in enumerate(w for w in widths if w <= WIDEST[layers]):
        h = min(w, 5 + 7 * (k % 4))
        wide = _lattice(layers, h + 2, w + 1, 1000 * layers + w, via_mask=k % 2 == 0)
        _check(wide, _nets(wide, w, h, 3, w))
        if w <= 2100:  # the transposed frame
            tall = _lattice(layers, w + 1, h + 2, 2000 * layers + w, via_mask=k % 2 == 1)
            _check(tall, _nets(tall, h, w, 3, w + 1))


@pytest.mark.parametrize("layers", [1, 4])
@pytest.mark.parametrize("costs", [(10, 25, 7), (10, 6, 3), (7, 7, 1), (400, 100, 9)])
def test_move_costs_on_both_sides_of_a_straight_move(layers, costs):
    lat = _lattice(layers, 90, 640, 5 + layers, True, costs)
    for w, h in ((70, 60), (300, 40), (600, 80)):
        _check(lat, _nets(lat, w, h, 6, w))


@pytest.mark.parametrize("layers", sorted(WIDEST))
def test_a_row_past_the_widest_shape_is_rejected(layers):
    w = WIDEST[layers] + 1
    lat = _lattice(layers, 3, w, 9, False)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        res, _ = dev.route(_nets(lat, w, 2, 2, 1), generator="sweep")
    finally:
        dev.close()
    assert (res["completion"] == apgar_b200.COMPLETION_REJECTED).all()
