"""The sweep's shapes for classes with more nets than the device has SMs, and
the rows where the shapes change, against the oracle (costs, canonical paths
and the schedule's counters are whole numbers and must be equal)."""

import pytest

from tests.test_lattice_sweep_shapes_gpu import WIDEST, _check, _lattice, _nets

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("layers", sorted(WIDEST))
def test_rows_where_the_shapes_change(layers):
    widths = [383, 384, 385, 640, 641, 1151, 1153, 1279, 1281, 1535, 1536, 1663, 1665, 1793, 1921, 2048, 2305, 3073,
              3585, 4607, 6145, 7681]
    for k, w in enumerate(w for w in widths if w <= WIDEST[layers]):
        h = min(w, 5 + 7 * (k % 4))
        wide = _lattice(layers, h + 2, w + 1, 3000 * layers + w, via_mask=k % 2 == 1)
        _check(wide, _nets(wide, w, h, 3, w))
        if w <= 2100:  # the transposed frame
            tall = _lattice(layers, w + 1, h + 2, 4000 * layers + w, via_mask=k % 2 == 0)
            _check(tall, _nets(tall, h, w, 3, w + 1))


@pytest.mark.parametrize("layers", sorted(WIDEST))
@pytest.mark.parametrize("width", [500, 513, 768, 769, 1024])
def test_a_class_with_more_nets_than_sms(layers, width):
    h = 6
    lat = _lattice(layers, 24, 1100, 5000 * layers + width, via_mask=width % 2 == 0)
    _check(lat, _nets(lat, width, h, _sms() + 5, width))
    tall = _lattice(layers, 1100, 32, 6000 * layers + width, via_mask=width % 2 == 1)
    _check(tall, _nets(tall, h, width, _sms() + 5, width + 1))
