"""The sweep's row width classes, on the CPU: the table in the kernel's source,
compiled by itself, covers every width without a gap, stays within a CTA, and
lets two nets share an SM wherever a batch may bring more of them than SMs."""

import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apgar_b200", "csrc")
WIDEST = {1: 8192, 2: 4096, 3: 2048, 4: 2048, 6: 1024, 8: 1024}
FIELDS = ("width", "cells", "warps", "most", "nets", "lanes")


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    with open(os.path.join(CSRC, "lattice_sweep.cu")) as f:
        rule = re.search(r"constexpr SweepShape row_lanes\(.*?\n(?=template <int L, int kIndex)", f.read(), re.S).group(0)
    with open(os.path.join(CSRC, "lattice_common.cuh")) as f:
        record = re.search(r"struct SweepShape \{.*?\};", f.read(), re.S).group(0)
    folder = tmp_path_factory.mktemp("shapes")
    source, program = str(folder / "shapes.cc"), str(folder / "shapes")
    with open(source, "w") as f:
        f.write("#include <cstdio>\n#include <initializer_list>\n" + record + "\n" + rule + """
int main() {
  for (int layers : {1, 2, 3, 4, 6, 8})
    for (int crowded = 0; crowded < 2; ++crowded)
      for (int i = 0;; ++i) {
        const SweepShape s = sweep_shape_at(layers, i, crowded != 0);
        if (s.width == 0) break;
        std::printf("%d %d %d %d %d %d %d %d\\n", layers, crowded, s.width, s.cells, s.warps, s.most, s.nets, s.lanes);
      }
}
""")
    subprocess.run(["g++", "-std=c++17", source, "-o", program], check=True)
    out = {}
    for line in subprocess.run([program], capture_output=True, text=True, check=True).stdout.splitlines():
        layers, crowded, *values = map(int, line.split())
        out.setdefault((layers, bool(crowded)), []).append(dict(zip(FIELDS, values)))
    return out


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("layers", sorted(WIDEST))
def test_classes_cover_every_width(tables, layers, crowded):
    table = tables[layers, crowded]
    assert [s["width"] for s in table] == sorted({s["width"] for s in tables[layers, False]})
    assert table[-1]["width"] == WIDEST[layers]
    for s in table:
        assert 32 * s["cells"] * s["warps"] == s["width"] and s["cells"] % 4 == 0 and s["cells"] <= 16
        # warps of a CTA, and the kernel's bound on them
        warps = s["most"] if s["lanes"] else s["most"] * layers
        assert s["warps"] <= s["most"] and warps <= 16
        # the registers that the bound leaves a thread, for the nets that an SM holds
        assert s["nets"] * 32 * warps * 64 <= 65536


def test_crowded_classes_leave_room_for_two_nets(tables):
    for layers in (2, 3, 4):
        for s in tables[layers, True]:
            if 512 < s["width"] <= 1024:
                assert s["lanes"] or s["nets"] >= 2, (layers, s)


def test_wide_rows_of_few_layers_take_the_form_with_fewer_barriers(tables):
    for layers, from_width in ((1, 1024), (2, 512)):
        for crowded in (False, True):
            assert all(bool(s["lanes"]) == (s["width"] > from_width) for s in tables[layers, crowded])
