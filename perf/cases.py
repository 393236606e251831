"""The calls whose speed is tracked: what users of this framework run, from the
smallest call to the largest batch.

Each case is one pass through a public entry point: lattice routing with both
generators (one-shot, resident and allocation-free), negotiated rip-up rounds,
learned corridors and their training, and the drop-in candidate batches in
both readback forms.  Inputs are seeded boards of the configurations in
``apgar_b200.synth`` and of the same ranges.

The frontier generator's work counters (rounds, expansions, levels) depend on
the order of concurrent relaxations and differ from run to run, so a frontier
pass returns every other field of its results; the sweep's counters follow
its schedule and are returned.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import apgar_b200
from apgar_b200 import dropin, learned, negotiate, prices, synth

GRID, ROWS = 64, 66  # the corridor network's coarse grid, and its padded rows
U64_MAX = (1 << 64) - 1


def listed():
    return [
        # a small board, every net searched over the whole board
        dict(name="route_small", kind="route", layers=2, height=256, width=256, blocked=0.20, nets=64,
             hpwl=0, sigma=0.0, via_mask=False, generator="frontier", validate=False),
        # a handful of nets rerouted on a larger board: latency counts
        dict(name="route_few", kind="route", layers=4, height=1024, width=1024, blocked=0.25, nets=8,
             hpwl=200, sigma=0.6, via_mask=False, generator="frontier", validate=False),
        # an odd board with via keep-outs and an odd number of nets
        dict(name="route_ragged", kind="route", layers=3, height=1000, width=1504, blocked=0.22, nets=777,
             hpwl=120, sigma=0.8, via_mask=True, generator="frontier", validate=False),
        # the medium benchmark batch from host buffers, every path validated
        dict(name="route_medium", kind="route", layers=4, height=2048, width=2048, blocked=0.25, nets=4096,
             hpwl=200, sigma=1.0, via_mask=False, generator="frontier", validate=True),
        # a resident plan of long nets on many layers, executed and read back
        dict(name="plan_long", kind="plan", layers=8, height=1536, width=1536, blocked=0.30, nets=200,
             hpwl=400, sigma=0.8, via_mask=False, generator="frontier"),
        # the plain sweep, the default generator
        dict(name="sweep_batch", kind="route", layers=4, height=1024, width=1024, blocked=0.25, nets=1024,
             hpwl=150, sigma=0.8, via_mask=False, generator="sweep", validate=False),
        # a planar board routed inside a process that must not allocate
        dict(name="noalloc_planar", kind="noalloc", layers=1, height=1024, width=1024, blocked=0.20, nets=96,
             hpwl=120, sigma=0.5, via_mask=False),
        # rip-up and reroute of multi-terminal nets, captured once as a graph
        dict(name="negotiate", kind="negotiate", layers=6, height=768, width=768, blocked=0.25, nets=800,
             hpwl=150, sigma=0.9, rounds=6, partial=True),
        # corridors proposed by the network, then the certified search
        dict(name="learned_route", kind="learned", layers=4, height=1536, width=1536, blocked=0.25, nets=1024,
             hpwl=200, sigma=0.9),
        # one training step of the corridor network: forward, backward, Adam
        dict(name="train_step", kind="train", nets=256, span=40),
        # alternative candidates on a compiled board, compact paths
        dict(name="dropin_compact", kind="dropin", side=26, bend=7, queries=64, workspace=False),
        # every heading state's label and predecessor on a board above the
        # shared-memory size
        dict(name="dropin_workspace", kind="dropin", side=48, bend=3, queries=16, workspace=True),
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["route", "route", "route", "plan", "sweep", "noalloc", "negotiate", "learned", "train",
                       "dropin"])
    if kind in ("route", "plan", "sweep"):
        layers = rng.choice([1, 2, 3, 4, 6, 8])
        top = 2048 if layers <= 4 else 1536
        height, width = _spread(rng, 200, top), 32 * _spread(rng, 7, top // 32)
        case = dict(kind="plan" if kind == "plan" else "route", layers=layers, height=height, width=width,
                    blocked=rng.choice([0.2, 0.25, 0.3]), nets=_spread(rng, 3, 1200),
                    hpwl=_spread(rng, 20, max(40, min(height, width) // 4)), sigma=rng.choice([0.5, 0.8, 1.0]),
                    via_mask=rng.random() < 0.4, generator="sweep" if kind == "sweep" else "frontier")
        if case["kind"] == "route":
            case["validate"] = rng.random() < 0.3
        return case
    if kind == "noalloc":
        return dict(kind="noalloc", layers=rng.choice([1, 2, 4]), height=_spread(rng, 256, 1024),
                    width=32 * _spread(rng, 8, 32), blocked=0.2, nets=_spread(rng, 4, 40),
                    hpwl=_spread(rng, 20, 80), sigma=0.4, via_mask=rng.random() < 0.4)
    if kind == "negotiate":
        size = 32 * _spread(rng, 10, 24)
        return dict(kind="negotiate", layers=rng.choice([2, 4, 6]), height=size, width=size, blocked=0.25,
                    nets=_spread(rng, 50, 700), hpwl=_spread(rng, 60, 150), sigma=0.8, rounds=rng.randint(2, 6),
                    partial=rng.random() < 0.7)
    if kind == "learned":
        return dict(kind="learned", layers=rng.choice([2, 4]), height=_spread(rng, 400, 1536),
                    width=32 * _spread(rng, 13, 48), blocked=0.25, nets=_spread(rng, 60, 1024),
                    hpwl=_spread(rng, 80, 200), sigma=0.8)
    if kind == "train":
        return dict(kind="train", nets=_spread(rng, 16, 256), span=rng.randint(20, 63))
    return dict(kind="dropin", side=rng.randint(9, 48), bend=rng.choice([0, 3, 7]), queries=_spread(rng, 4, 128),
                workspace=rng.random() < 0.3)


# ------------------------------- inputs ------------------------------------

def _board(case, seed):
    """The case's lattice: a seeded square one, cut to height x width."""
    size = -(-max(case["height"], case["width"]) // 32) * 32
    pads = case["layers"] > 2
    lat = synth.make_lattice(seed, case["layers"], size, case["blocked"], pads=pads,
                             via_mask=case.get("via_mask", False))
    if (case["height"], case["width"]) == (size, size):
        return lat
    cut = lambda a: None if a is None else np.ascontiguousarray(a[:, :case["height"], :case["width"] // 32])  # noqa: E731
    return synth.Lattice(lat.layers, case["height"], case["width"], cut(lat.blocked), cut(lat.via_ok))


def _nets(case, lat, seed):
    if case["kind"] == "negotiate":  # about three segments a net: the first two a net on average
        segments, _ = synth.make_multi_terminal_nets(lat, seed + 1, case["nets"], float(case["hpwl"]), case["sigma"])
        return np.ascontiguousarray(np.resize(segments, 2 * case["nets"]))
    if case["hpwl"] == 0:
        return synth.make_nets(lat, seed + 1, case["nets"], hpwl_median=None, margin=None)
    many = case["nets"] * (4 if case["kind"] == "noalloc" else 1)
    nets = synth.make_nets(lat, seed + 1, many, hpwl_median=float(case["hpwl"]), hpwl_sigma=case["sigma"])
    if case["kind"] == "noalloc":
        # the caller sends the nets that fit the fixed scratch together
        need = 4 * synth.window_cells(lat, nets) + 8 * (8 * (nets["win_w"].astype(np.int64) + nets["win_h"]) + 64 * lat.layers)
        nets = np.resize(nets[need < apgar_b200.NOALLOC_SCRATCH_BYTES * 3 // 4 // case["nets"]], case["nets"])
    return np.ascontiguousarray(nets)


def _path_cells(case):
    """Room for every path of the batch, in the caller's own buffer."""
    if case["kind"] == "dropin":
        return case["queries"] * 9 * case["side"] ** 2
    count = case["nets"] * (2 if case["kind"] == "negotiate" else 1)
    return int(4 * count * (_span(case) + 100))


def _span(case):
    """Mean half-perimeter of the case's nets, in cells."""
    if case["hpwl"] == 0:
        return 0.52 * (case["height"] + case["width"])
    return case["hpwl"] * math.exp(case["sigma"] ** 2 / 2)


NODE_DTYPE = np.dtype([("lattice_x", "<i8"), ("lattice_y", "<i8"), ("layer", "<u4"), ("legal_edges", "u1"),
                       ("reserved", "u1", (3,)), ("neighbors", "<u4", (8,))])
RUN_DTYPE = np.dtype([("node_offset", "<u4"), ("node_count", "<u4"), ("direction", "u1"), ("reserved", "u1", (3,))])
LAYER_DTYPE = np.dtype([("layer", "<u4"), ("node_offset", "<u4"), ("node_count", "<u4"), ("padding", "<u4"),
                        ("minimum_lattice_x", "<i8"), ("maximum_lattice_x", "<i8"), ("minimum_lattice_y", "<i8"),
                        ("maximum_lattice_y", "<i8")])
STEPS = ((1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0), (-1, -1), (0, -1), (1, -1))


def _compiled_board(side, bend, rng):
    """A side x side compiled board with wall segments cut out of its edges."""
    cut = np.zeros((side, side), bool)
    for _ in range(side // 3):
        x, y = (int(v) for v in rng.integers(1, side - 1, size=2))
        if rng.integers(2):
            cut[y, max(0, x - side // 4):x + side // 4] = True
        else:
            cut[max(0, y - side // 4):y + side // 4, x] = True
    n = side * side
    ys, xs = np.divmod(np.arange(n), side)
    nodes = np.zeros(n, NODE_DTYPE)
    nodes["lattice_x"], nodes["lattice_y"], nodes["neighbors"] = xs, ys, 0xFFFFFFFF
    legal = np.zeros((8, n), bool)
    for d, (dx, dy) in enumerate(STEPS):
        nx, ny = xs + dx, ys + dy
        inside = (nx >= 0) & (nx < side) & (ny >= 0) & (ny < side)
        legal[d] = inside & ~cut.ravel() & ~cut[np.clip(ny, 0, side - 1), np.clip(nx, 0, side - 1)]
        nodes["neighbors"][:, d] = np.where(legal[d], ny * side + nx, 0xFFFFFFFF)
    nodes["legal_edges"] = (legal * (1 << np.arange(8))[:, None]).sum(0)
    runs, run_nodes = [], []
    for d, (dx, dy) in enumerate(STEPS):
        for i in np.flatnonzero(legal[d] & ~legal[(d + 4) % 8]):
            chain = [int(i)]
            while legal[d][chain[-1]]:
                chain.append(chain[-1] + dy * side + dx)
            runs.append((len(run_nodes), len(chain), d, (0, 0, 0)))
            run_nodes.extend(chain)
    run = np.array(runs, dtype=RUN_DTYPE)
    layers = np.zeros(1, LAYER_DTYPE)
    layers["node_count"], layers["maximum_lattice_x"], layers["maximum_lattice_y"] = n, side - 1, side - 1
    h = np.zeros(1, dropin.HEADER_DTYPE)
    h["schema_version"], h["compiler_version"], h["represented_nodes"], h["represented_states"] = 1, 1, n, 9 * n
    h["lattice_step"], h["orthogonal_step"], h["diagonal_step"], h["bend"], h["heading_mask"] = 1, 10, 14, bend, 7
    h["estimated_persistent_device_bytes"] = 112 + 48 + 56 * n + 12 * len(run) + 4 * len(run_nodes)
    return (h, layers, nodes, run, np.array(run_nodes, np.uint32)), cut, legal


def _candidates(case, rng, cut, legal):
    """Alternative candidates: plain, surcharged, and with edge policies."""
    free, diagonal = np.flatnonzero(~cut.ravel()), np.flatnonzero(legal[1])
    entries = []
    for i in range(case["queries"]):
        s, g = rng.choice(free, size=2, replace=False)
        e = dict(start_node=int(s), goal_node=int(g))
        if i % 3 == 1:
            e.update(orthogonal_step_surcharge=2, bend_surcharge=5)
        if i % 3 == 2:
            picks = np.sort(rng.choice(diagonal, size=min(12, len(diagonal)), replace=False))
            policy = np.zeros(len(picks), dropin.POLICY_EDGE_DTYPE)
            policy["physical_edge_index"], policy["adjustment"] = picks.astype(np.uint32) * 8 + 1, 40
            policy["adjustment"][:2] = U64_MAX
            e.update(policy=policy)
        entries.append(e)
    return entries


def _training_batch(case, seed):
    """Coarse rasters, window sizes, path labels and weights as host arrays."""
    rng = np.random.default_rng(seed)
    n = case["nets"]
    cw = np.clip(np.rint(case["span"] * np.exp(0.4 * rng.standard_normal(n))), 17, 63).astype(np.int64)
    ch = np.clip(np.rint(case["span"] * np.exp(0.4 * rng.standard_normal(n))), 17, 63).astype(np.int64)
    mask = (np.arange(GRID)[None, None, :] < cw[:, None, None]) & (np.arange(GRID)[None, :, None] < ch[:, None, None])
    raster = np.zeros((n, ROWS, GRID, 16), np.float32)
    inner = raster[:, 1:GRID + 1]
    inner[..., :4] = np.clip(rng.normal(0.25, 0.2, (n, GRID, GRID, 4)), 0, 1)
    inner[..., 4:10] = rng.random((n, 1, 1, 6))
    inner[..., 10:14] = (np.arange(GRID) / GRID)[None, None, :, None]
    labels = np.zeros((n, GRID, GRID), np.uint8)
    for i in range(n):
        x0, x1 = sorted(int(v) for v in rng.integers(0, cw[i], size=2))
        y0, y1 = (int(v) for v in rng.integers(0, ch[i], size=2))
        t = np.linspace(0, 1, 2 * GRID)
        labels[i, np.rint(y0 + t * (y1 - y0)).astype(int), np.rint(x0 + t * (x1 - x0)).astype(int)] = 1
        inner[i, y0, x0, 14] = inner[i, y1, x1, 15] = 1
    inner *= mask[..., None]
    dims = (cw | (ch << 8) | (2 << 16)).astype(np.uint32)
    parts = []
    for layer in range(5):
        cin = 16 if layer == 0 else 32
        parts += [rng.normal(0, math.sqrt(2 / (9 * cin)), 32 * 9 * cin), 0.01 * rng.standard_normal(32)]
    parts += [rng.normal(0, math.sqrt(1 / (9 * 32)), 9 * 32), np.array([-3.0])]
    return raster, dims, labels, np.concatenate(parts).astype(np.float32), mask


# --------------------------- prepare, run, work ----------------------------

def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "train":
        raster, dims, labels, weights, _ = _training_batch(case, seed)
        net = learned.CorridorNet(weights)
        state.update(net=net, weights=torch.from_numpy(weights).cuda(),
                     rasters=torch.from_numpy(raster).cuda().to(torch.bfloat16), dims=torch.from_numpy(dims).cuda(),
                     labels=torch.from_numpy(labels).cuda(), acts=net.activations(case["nets"], distinct=True))
        return state
    if kind == "dropin":
        rng = np.random.default_rng(seed)
        records, cut, legal = _compiled_board(case["side"], case["bend"], rng)
        view = dropin.View(*records)
        generator = dropin.GENERATOR_FRONTIER if case["workspace"] else dropin.GENERATOR_PERSISTENT
        queries, edges = dropin.make_queries(view.node_count, _candidates(case, rng, cut, legal), generator=generator)
        state.update(view=view, queries=queries, edges=edges, generator=generator,
                     paths=np.zeros(_path_cells(case), np.uint32))
        return state
    lat = _board(case, seed)
    nets = _nets(case, lat, seed)
    dev = apgar_b200.DeviceLattice(lat)
    # the caller's result buffers, pinned and kept from call to call
    results = torch.zeros(len(nets) * apgar_b200.RESULT_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy()
    paths = torch.zeros(_path_cells(case), dtype=torch.int32).pin_memory().numpy()
    state.update(dev=dev, nets=nets, results=results.view(apgar_b200.RESULT_DTYPE), paths=paths.view(np.uint32))
    if kind in ("plan", "negotiate", "learned"):
        state["plan"] = dev.plan(nets, generator="frontier")
    if kind == "negotiate":
        state["negotiation"] = negotiate.Negotiation(state["plan"], prices.policy(capacity=1))
    if kind == "learned":
        state["router"] = learned.LearnedRouter(state["plan"])
    return state


def _kept(state, paths):
    """Paths read back, in the caller's own buffer."""
    state["paths"][:len(paths)] = paths
    return state["paths"]


def _routes(state, results, paths, counters):
    names = ["cost", "completion", "path_len", "path_offset"]
    names += ["sweeps", "row_steps", "row_stores", "row_loads"] if counters else []
    if not np.shares_memory(paths, state["paths"]):
        _kept(state, paths)
    return {**{k: results[k] for k in names}, "paths": state["paths"]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "route":
        results, paths = state["dev"].route(state["nets"], generator=case["generator"],
                                            out=(state["results"], state["paths"]))
        out = _routes(state, results, paths, case["generator"] == "sweep")
        if case["validate"]:
            verdicts = state["dev"].validate(state["nets"], results, paths)
            out.update({k: verdicts[k] for k in ("code", "failing_index", "total_cost")})
        return out
    if kind == "plan":
        state["plan"].execute()
        return _routes(state, *state["plan"].readback(), False)
    if kind == "noalloc":
        return _routes(state, *state["dev"].route_noalloc(state["nets"], out=(state["results"], state["paths"])), True)
    if kind == "negotiate":
        n = state["negotiation"]
        n.run(case["rounds"], use_graph=True, partial=case["partial"])
        usage, history, costs, stats = n.readback()
        out = _routes(state, *state["plan"].readback(), False)
        out.update(usage=usage, history=history, costs=costs,
                   stats=np.array([[s["overused_cells"], s["total_overuse"], s["price_status"]] for s in stats]))
        return out
    if kind == "learned":
        state["router"].execute()
        out = _routes(state, *state["plan"].readback(), False)
        out["status"] = state["plan"].corridor_status()
        return out
    if kind == "train":
        # each pass is the first step from the state's own weights
        net = state["net"]
        net.params.copy_(state["weights"])
        net.m.zero_()
        net.v.zero_()
        net.step = 0
        net.prepare()
        loss = net.train_step(state["rasters"], state["dims"], state["labels"], lr=1e-3, acts=state["acts"])
        return {"loss": loss, "grads": net.grads, "params": net.params}
    pending = state["view"].execute_batch(state["queries"], state["edges"], generator=state["generator"])
    results, compact, states, _ = pending.readback()
    out = {k: results[k] for k in ("goal_state", "completion", "query_id")}
    out.update(state_count=compact["state_count"], state_offset=compact["state_offset"], states=_kept(state, states))
    if case["workspace"]:
        out["labels"], out["predecessors"], out["owners"], out["predecessor_owners"] = pending.readback_workspace()
    pending.close()
    return out


def work(case):
    kind, n = case["kind"], case.get("nets", 0)
    if kind == "train":
        # forward, input gradient (layers 2-5) and weight gradient over the window cells
        cells = n * case["span"] ** 2
        first, rest = 9 * 16 * 32, 4 * 9 * 32 * 32
        return dict(bytes=cells * (16 * 2 + 1) + 4 * 7 * 42209, flops=2.0 * cells * (2 * first + 3 * rest))
    if kind == "dropin":
        nodes, q = case["side"] ** 2, case["queries"]
        per_query = 120 + 120 + 32 + 4 * case["side"] + (9 * nodes * 28 if case["workspace"] else 0)
        return dict(bytes=33 * nodes + q * per_query, flops=0)
    cells = case["layers"] * case["height"] * case["width"]
    records = n * (40 + 48 + 4 * 0.8 * _span(case))  # net, result, and a path of about this many cells
    total = cells / 8 * (2 if case.get("via_mask") else 1) + records
    if kind == "negotiate":
        total += 16 * cells + records  # usage, history and prices; two segments a net
    if case.get("validate"):
        total += records + 24 * n
    return dict(bytes=total, flops=0)


# ------------------------------ exact values -------------------------------

def exact(case, seed):
    """The training step in 64 bits; the other outputs are whole numbers."""
    if case["kind"] != "train":
        return None
    raster, dims, labels, weights, mask = _training_batch(case, seed)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.from_numpy(raster[:, 1:GRID + 1]).to(torch.bfloat16).to(device, torch.float64).permute(0, 3, 1, 2)
    m = torch.from_numpy(mask).to(device, torch.float64)
    flat = torch.from_numpy(weights).to(device, torch.float64).requires_grad_()
    at, a = 0, x

    def conv(v, w):  # w [out][tap][in], tap = (dy + 1) * 3 + dx + 1
        padded = torch.nn.functional.pad(v, (1, 1, 1, 1))
        return sum(torch.einsum("nchw,oc->nohw", padded[:, :, t // 3:t // 3 + GRID, t % 3:t % 3 + GRID], w[:, t])
                   for t in range(9))

    for layer in range(5):
        cin = 16 if layer == 0 else 32
        w, at = flat[at:at + 32 * 9 * cin].view(32, 9, cin), at + 32 * 9 * cin
        b, at = flat[at:at + 32], at + 32
        a = torch.relu(conv(a, w) + b[None, :, None, None]) * m[:, None]
    w, at = flat[at:at + 288].view(1, 9, 32), at + 288
    z = conv(a, w)[:, 0] + flat[at]
    t = torch.from_numpy(labels).to(device, torch.float64)
    weight = torch.where(t > 0, 8.0, 1.0) * m / (m.sum((1, 2), keepdim=True) * len(labels))
    loss = (weight * torch.nn.functional.binary_cross_entropy_with_logits(z, t, reduction="none")).sum()
    loss.backward()
    g = flat.grad
    # Adam's first step: both moments are bias-corrected to g and g * g
    params = flat.detach() - 1e-3 * g / (g.abs() + 1e-8)
    return {"loss": loss.detach().reshape(1), "grads": g, "params": params}
