"""Batches of small windows: the form of the search is chosen by the number of
nets, their windows and the layers, and results do not depend on it.  Costs and
canonical paths are whole numbers and must equal the oracle's; priced ones must
equal those of the search over cells."""

import numpy as np
import pytest

import apgar_b200
import oracle
from apgar_b200 import negotiate, prices, synth
from tests.test_lattice_tiles_gpu import CELL_FORM, _windows
from tests.test_tile_slots_gpu import _words

pytestmark = pytest.mark.gpu

# layers, window, nets, whether an unpriced search takes the tiles
CASES = [(1, 16, 16, 64, False), (1, 16, 16, 65, True), (1, 17, 16, 64, True), (3, 4, 4, 24, False),
         (8, 128, 128, 4, False), (8, 128, 129, 4, True), (8, 128, 128, 5, True), (6, 40, 40, 4, True),
         (8, 181, 181, 40, True), (8, 182, 181, 12, True), (4, 101, 101, 32, True), (4, 101, 102, 32, True),
         (4, 100, 100, 33, True)]


@pytest.mark.parametrize("layers,w,h,count,tiles", CASES)
def test_results_do_not_depend_on_the_form(layers, w, h, count, tiles):
    import torch

    lat = synth.make_lattice(600 + layers, layers, 256, 0.2, via_mask=layers > 1)
    nets = _windows(lat, w, h, count, w + h + count)
    rng = np.random.default_rng(601)
    cells = layers * 256 * 256
    costs = torch.from_numpy(np.where(rng.random(cells) < 0.1, rng.integers(1, 400, cells), 0).astype(np.int32)).cuda()
    exact, paths_o = oracle.dijkstra_batch(lat, nets)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        plans = [dev.plan(nets, generator="frontier"), dev.plan(nets, generator="frontier", max_rounds=CELL_FORM)]
        assert (plans[0].info()["label_cells"] == sum(_words(lat, n) for n in nets)) == tiles
        out = []
        for plan in plans:
            for prices_now in (None, costs, None, costs):
                plan.set_cell_costs(prices_now)
                plan.execute()
                res, paths = plan.readback()
                out.append((res["cost"].copy(), res["completion"].copy(), paths.copy()))
                if prices_now is None:
                    assert np.array_equal(res["cost"], exact)
                    for mine, theirs, cost in zip(apgar_b200.split_paths(res, paths), paths_o, exact):
                        assert cost == oracle.lo_inf() or np.array_equal(mine, theirs)
        for a, b in zip(out[:4], out[4:]):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))
        rounds = []
        for plan in plans:
            plan.set_cell_costs(None)
            n = negotiate.Negotiation(plan, prices.policy(capacity=1))
            n.run(4, use_graph=True, partial=True)
            rounds.append([x for x in n.readback()[:3]] + [plan.readback()[1]])
            n.close()
            plan.close()
        assert all(np.array_equal(x, y) for x, y in zip(*rounds))
        res, _ = dev.route(nets, generator="frontier")
        assert np.array_equal(res["cost"], exact)
    finally:
        dev.close()


def test_a_large_batch_of_small_nets_does_not_wait_for_the_host():
    """5,000 more nets of one unit take less than 0.5 us more each: a read of the
    host's cancel flag at every start takes about 1 us, one after the other."""
    import torch

    lat = synth.make_lattice(611, 1, 512, 0.1)
    nets = _windows(lat, 12, 12, 6000, 612)
    dev = apgar_b200.DeviceLattice(lat)
    try:
        stream = torch.cuda.current_stream().cuda_stream
        best = []
        for batch in (nets[:1000], nets):
            plan = dev.plan(batch, generator="frontier")
            times = []
            for _ in range(8):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                plan.execute(stream)
                b.record()
                b.synchronize()
                times.append(a.elapsed_time(b))
            best.append(min(times[1:]))
            plan.close()
    finally:
        dev.close()
    assert 1e3 * (best[1] - best[0]) < 0.5 * 5000, best
