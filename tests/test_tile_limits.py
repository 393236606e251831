"""The tile search's guards, on the CPU: how many passes a unit can need, that
a unit at its limit ends before a waiting owner loses patience, and that a slot
whose net was given up is not handed to another net."""

import os
import re

import numpy as np
import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apgar_b200", "csrc",
                      "lattice_tiles.cu")
INF = 1 << 30
ORTH, DIAG = 10, 14


def _constant(name):
    with open(SOURCE) as f:
        value = re.search(rf"\b{name} = (?P<v>1u? << \d+);", f.read())["v"]
    return 1 << int(value.split("<<")[1])


def _passes(free, start):
    """Passes over a unit until nothing changes: each a sweep down, up, right
    and left, a line taking the straight and both diagonal moves from the last."""
    label = np.full((32, 32), INF)
    label[start] = 0
    passes = 0
    while True:
        passes += 1
        before = label.copy()
        for grid, open_ in ((label, free), (label[::-1], free[::-1]), (label.T, free.T), (label.T[::-1], free.T[::-1])):
            for i in range(1, 32):
                src, dst = open_[i - 1], open_[i]
                best = np.where(dst, grid[i - 1] + ORTH, INF)
                both = src & dst  # side cells of the diagonals
                best[1:] = np.minimum(best[1:], np.where(both[1:] & both[:-1], grid[i - 1, :-1] + DIAG, INF))
                best[:-1] = np.minimum(best[:-1], np.where(both[:-1] & both[1:], grid[i - 1, 1:] + DIAG, INF))
                grid[i] = np.minimum(grid[i], best)
        if np.array_equal(label, before):
            return passes, label


def _serpentine():
    free = np.zeros((32, 32), bool)
    free[0::2] = True
    free[1::4, 31] = free[3::4, 0] = True
    return free


def _staircase_serpentine():
    """One-cell corridors that turn at every second cell."""
    free = np.zeros((32, 32), bool)
    y = 0
    while y + 2 < 32:
        for x in range(0, 31, 4):
            free[y, x:x + 3] = True
            free[y:y + 3, x + 2] = True
            free[y + 2, x + 2:x + 5] = True
            free[y:y + 3, min(x + 4, 31)] = True
        y += 4
        if y < 32:
            free[y - 2:y + 1, 30 if (y // 4) % 2 else 0] = True
    return free


def _spiral():
    free = np.zeros((32, 32), bool)
    y, x, dy, dx = 0, 0, 0, 1
    free[0, 0] = True
    for length in (31, 31, 31, 29, 29, 27, 27, 25, 25, 23, 23, 21, 21, 19, 19, 17, 17, 15, 15, 13, 13, 11, 11, 9, 9, 7, 7, 5, 5, 3, 3):
        for _ in range(length):
            if not (0 <= y + dy < 32 and 0 <= x + dx < 32):
                break
            y, x = y + dy, x + dx
            free[y, x] = True
        dy, dx = dx, -dy
    return free


def _tree(seed):
    """A random maze: a spanning tree over every second cell."""
    rng = np.random.default_rng(seed)
    free = np.zeros((32, 32), bool)
    free[0, 0] = True
    stack = [(0, 0)]
    while stack:
        y, x = stack[-1]
        steps = [(dy, dx) for dy, dx in ((0, 2), (2, 0), (0, -2), (-2, 0))
                 if 0 <= y + dy < 31 and 0 <= x + dx < 31 and not free[y + dy, x + dx]]
        if not steps:
            stack.pop()
            continue
        dy, dx = steps[rng.integers(len(steps))]
        free[y + dy // 2, x + dx // 2] = free[y + dy, x + dx] = True
        stack.append((y + dy, x + dx))
    return free


@pytest.mark.parametrize("maze", [_serpentine, _staircase_serpentine, _spiral, lambda: _tree(1), lambda: _tree(2),
                                  lambda: np.ones((32, 32), bool)])
def test_a_unit_needs_fewer_passes_than_its_limit(maze):
    free = maze()
    passes, label = _passes(free, (0, 0))
    assert (label < INF).sum() > 100
    assert passes <= 1024 < _constant("kMaxUnitPasses")


def test_a_unit_at_its_limit_ends_before_an_owner_gives_up():
    # cycles: 4 sweeps of 32 steps a pass, 6 warps on each quarter of the SM,
    # against three dependent reads of the L2 at 250 cycles or more a look
    longest = _constant("kMaxUnitPasses") * 128 * 34 * 6
    patience = _constant("kIdleLimit") * 3 * 250
    assert longest < patience


def test_a_slot_with_a_warp_left_in_it_takes_no_other_net():
    with open(SOURCE) as f:
        kernel = f.read().split("lattice_tiles_kernel(const __grid_constant__ TileLaunch p) {")[1]
    given_up = kernel.index("*reinterpret_cast<volatile uint32_t*>(p.finished + 1) = 1u;")
    assert kernel.index("atomicMax(&st->stop, 2u)") < given_up < kernel.index("finish_net<kPriced>")
    guard = kernel.index("p.per_net == 0u && __shfl_sync(kFull, peek(p.finished + 1), 0) != 0u")
    assert kernel.index("reject_net(st, lane)", guard) < kernel.index("start_net(p, n, st", guard)
    assert kernel.count("start_net(") == 1
