"""Order of a tile unit's announcements, explored on the CPU.

A warp that has relaxed a unit stores its labels, marks the unit as labelled,
sets its side bit in the neighbours it lowers, lowers their keys, and frees its
own key.  Another warp may take a neighbour, or the unit itself, between any
two of these.  The test reads the sequence and its fences from the kernel's
source, generates every order in which the memory accesses may land, places
the other warp everywhere in it, and requires that no lowering is lost."""

import itertools
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apgar_b200", "csrc",
                      "lattice_tiles.cu")
TOKENS = {
    "labels": r"mine\[\(c \+ k\) \* 32\] = v;",
    "touched": r"atomicOr\(ws\.flags \+ u\.id, kTouched\)",
    "side": r"atomicOr\(ws\.flags \+ nb, part\.seen\)",
    "key": r"atomicMin\(ws\.pend \+ nb, out_key\)",
    "free": r"finish\(near, far, packed \+ part\.packed\)",
    "branch": r"if \((?:out_key <= limit|lowers)\) \{",  # the lanes that go on to lower a neighbour
    "fence": r"__threadfence\(\)",
    "warp": r"__syncwarp\(\)",
}
LANES = {"labels": "all", "touched": "lane 0", "side": "neighbour lanes", "key": "neighbour lanes", "free": "lane 31"}


def _sequence():
    """The kernel's steps from the label stores to the end of the unit."""
    with open(SOURCE) as f:
        text = f.read()
    start = text.index("// changed rows (all of them the first time)")
    text = text[start:text.index("// Canonical reverse path by one warp", start)]
    text = re.sub(r"//[^\n]*", "", text)
    found = sorted((m.start(), name) for name, pattern in TOKENS.items() for m in re.finditer(pattern, text))
    steps, lowering = [], False
    for _, name in found:
        lowering = (lowering or name == "branch") and name != "free"
        # a fence inside the neighbours' branch is only those lanes'
        steps.append("own fence" if name == "fence" and lowering else name)
    steps = [s for s in steps if s != "branch"]
    assert [s for s in steps if s in LANES] == ["labels", "touched", "side", "key", "free"]
    return steps


def _side_bit_says_labelled():
    """Whether a warp reads a neighbour's labels on the side bit alone."""
    with open(SOURCE) as f:
        return "touched_neighbours(ws, part, u.id, exist, lane) | (flags & exist)" in f.read()


def _ordered(steps, a, b):
    """Whether access a lands before access b in every execution."""
    between = steps[steps.index(a) + 1:steps.index(b)]
    if LANES[a] == LANES[b]:
        return "fence" in between or "own fence" in between
    # from lane to lane: the lanes meet, and a fence of the whole warp
    return "fence" in between and "warp" in between


def _landings(steps):
    names = [s for s in steps if s in LANES]
    before = [(a, b) for a, b in itertools.combinations(names, 2) if _ordered(steps, a, b)]
    for order in itertools.permutations(names):
        if all(order.index(a) < order.index(b) for a, b in before):
            yield order


def _neighbour_is_lowered(order, taken_at, side_suffices):
    """The neighbour's warp takes its unit (queued by a third warp) before the
    access at index taken_at lands, and again whenever its key is lowered."""
    landed, side, entered = set(), False, False

    def take():
        nonlocal side, entered
        entered = entered or (side and "labels" in landed and (side_suffices or "touched" in landed))
        side = False

    for i, access in enumerate(order):
        if i == taken_at:
            take()
        landed.add(access)
        side = side or access == "side"
        if access == "key":
            take()
    return entered


def test_no_lowering_is_lost():
    orders = list(_landings(_sequence()))
    assert orders
    for order in orders:
        for taken_at in range(len(order) + 1):
            assert _neighbour_is_lowered(order, taken_at, _side_bit_says_labelled()), (order, taken_at)


def test_the_units_next_owner_sees_its_labels():
    for order in _landings(_sequence()):
        assert order.index("free") > max(order.index("labels"), order.index("touched")), order


def test_labels_land_before_they_are_announced():
    for order in _landings(_sequence()):
        assert order.index("labels") < min(order.index("touched"), order.index("side")), order


def test_the_model_finds_a_lost_lowering():
    # side bit and mark in either order, and a reader that waits for the mark
    steps = ["labels", "fence", "warp", "touched", "side", "own fence", "key", "warp", "free"]
    found = {side_suffices: all(_neighbour_is_lowered(order, at, side_suffices) for order in _landings(steps)
                                for at in range(len(order) + 1)) for side_suffices in (False, True)}
    assert found == {False: False, True: True}
