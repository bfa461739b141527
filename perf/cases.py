"""Workloads of the placement engine, through its public entry points.

Each case is one call (or the short sequence of calls) that a program using
the engine makes again and again:

  place     start positions restored, ep_initialize, a bounded
            ep_nesterov_run, the positions read back: the optimizer loop
  gradient  ep_set_positions, ep_eval_gradient, ep_get_gradient: a driver
            that owns its optimizer and asks for the placer's gradient
  qp        ep_quadratic_placement from the core centre, positions read back
  start     the learned start: the network's proposal on a netlist it has not
            seen, then the refinement round that the committed weights name
  train     the loss and weight gradient of one training design, its graph and
            features built anew as a step over many designs meets them
  batch     many small designs placed together (ep_run_batch)
  scatter   ep_density_scatter_noalloc on device arrays

Designs follow the generators of eplace_b200.synth (cell widths, power-law net
degrees, Rent-style locality, pads on a ring, macros), drawn here without
per-net Python loops.  Positions are a point between the core centre and a
cell's home in the cluster hierarchy, plus jitter: the clumped starts and the
spread placements that an optimizer run passes through.
"""
import ctypes
import math

import numpy as np
import torch

from eplace_b200 import placer, synth, warmstart

MEAN_DEGREE, MAX_DEGREE, RENT_P, LEAF = 3.6, 500, 0.6, 8
MACRO, FILLER = 1, 2  # flag bits of ep_density_scatter_noalloc
_F32P, _F64P = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_double)


# ---------------------------------------------------------------- the cases --
def listed():
    return [
        # the smallest design of the repository: 100 cells, 16 x 16 bins;
        # every launch and every host round trip counts
        dict(name="place_smoke", kind="place", cells=100, macros=0, bins=16, spread=0.5, steps=16),
        # a ragged mixed-size design with the Barzilai-Borwein step: macros
        # take the block-per-object paths, fixed macros the static maps
        dict(name="place_mixed_30k", kind="place", cells=30011, macros=24, bins=0, spread=0.7, steps=16, rule="bb"),
        # the benchmark's size: 200k cells, 512 x 512 bins, from a
        # partly spread start
        dict(name="place_200k", kind="place", cells=200_000, macros=0, bins=512, spread=0.6, steps=16),
        # the same loop in the plain FP64 form, from a clumped start
        dict(name="place_200k_fp64", kind="place", cells=200_000, macros=0, bins=512, spread=0.3, steps=16, fp64=True),
        # the largest: 1M cells with 300 macros on 1024 x 1024 bins
        dict(name="place_1m", kind="place", cells=1_000_000, macros=300, bins=1024, spread=0.8, steps=16),
        # one gradient of a small design with the other wirelength model and
        # the exact exponential
        dict(name="gradient_5k_lse", kind="gradient", cells=5003, macros=6, bins=0, spread=0.8, lse=True, exact_exp=True),
        # one gradient on a bin grid that is no power of two: the dense
        # transforms on the tensor cores
        dict(name="gradient_60k_384", kind="gradient", cells=60_000, macros=0, bins=384, spread=0.9),
        # the reference flow's start of the benchmark design: seven rounds
        dict(name="qp_200k", kind="qp", cells=200_000, rounds=7),
        # the learned start of the benchmark design
        dict(name="start_200k", kind="start", cells=200_000),
        # one training design at the top of the training range
        dict(name="train_50k", kind="train", cells=50_000),
        # small designs placed together, 2k to 16k cells
        dict(name="batch_16", kind="batch", designs=16, cells=2_000, top=16_000, steps=16),
        # the scatter for callers that bring their own memory
        dict(name="scatter_300k", kind="scatter", cells=300_000, bins=512, spread=0.8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["place", "place", "place", "gradient", "gradient", "qp", "start", "train", "batch", "scatter"])
    if kind == "place":
        fp64 = rng.random() < 0.25
        cells = _log_int(rng, 300, 300_000 if fp64 else 600_000)
        bins = rng.choice([0, 0, 0, 2 ** max(4, min(10, round(math.log2(cells) / 2) + rng.choice([-1, 0]))),])
        return dict(kind=kind, cells=cells, macros=rng.choice([0, 0, rng.randint(2, 60)]) if cells > 2000 else 0,
                    bins=bins, spread=round(rng.uniform(0.2, 1.0), 3), steps=rng.choice([6, 8, 13, 16, 24]), fp64=fp64,
                    rule=rng.choice(["lipschitz", "lipschitz", "bb"]), lse=rng.random() < 0.2)
    if kind == "gradient":
        return dict(kind=kind, cells=_log_int(rng, 200, 100_000), macros=rng.choice([0, rng.randint(2, 20)]),
                    bins=rng.choice([0, 0, 128, 200, 256, 384]), spread=round(rng.uniform(0.3, 1.0), 3),
                    lse=rng.random() < 0.3, exact_exp=rng.random() < 0.3, fp64=False)
    if kind == "qp":
        return dict(kind=kind, cells=_log_int(rng, 500, 200_000), rounds=rng.randint(2, 7))
    if kind == "start":
        return dict(kind=kind, cells=_log_int(rng, 2_000, 300_000))
    if kind == "train":
        return dict(kind=kind, cells=_log_int(rng, 2_000, 50_000))
    if kind == "batch":
        lo = _log_int(rng, 500, 4_000)
        return dict(kind=kind, designs=rng.randint(2, 20), cells=lo, top=lo * rng.randint(2, 8), steps=rng.choice([8, 13, 16]))
    return dict(kind=kind, cells=_log_int(rng, 500, 500_000), bins=rng.choice([64, 128, 200, 256, 512]),
                spread=round(rng.uniform(0.2, 1.0), 3))


# -------------------------------------------------------------- the designs --
def _home(idx, n):
    """Place of cell idx (of n) in the unit square: its index read as a Morton
    code, so that each cluster of the index order has a compact region."""
    code = ((idx + 0.5) / n * (1 << 20)).astype(np.int64)
    x = np.zeros(code.shape)
    y = np.zeros(code.shape)
    for b in range(10):
        x += ((code >> (2 * b + 1)) & 1) * 2.0 ** (b - 10)
        y += ((code >> (2 * b)) & 1) * 2.0 ** (b - 10)
    return x + 2.0 ** -11, y + 2.0 ** -11


def _netlist(rng, cells, macros=0, bins=0, utilisation=0.7):
    """A standard-cell design (synth.standard_cell's distributions, every cell
    on a net, pads near their cluster) with `macros` movable and macros // 6
    fixed macros; returns (synth.Netlist, home x, home y of the nodes)."""
    nc, nn, nt = cells, round(1.1 * cells), max(4, cells // 100)
    # the sizes in the design depend on the case alone, so that every seed has
    # the same number of fillers; which cell has which is the seed's
    sizes = np.random.default_rng([cells, macros])
    w = rng.permutation(np.clip(np.rint(sizes.lognormal(math.log(3.0) - 0.18, 0.6, nc)), 1, 20))
    base_side = math.sqrt(w.sum() / utilisation)
    nf = macros // 6
    ms = np.maximum(np.rint(np.exp(sizes.uniform(math.log(0.01 * base_side + 2), math.log(0.05 * base_side + 3), macros + nf))), 2)
    mw = ms * np.where(sizes.random(macros + nf) < 0.5, 1.0, 2.0)
    side = float(math.ceil(math.sqrt((w.sum() + (mw * ms).sum()) / utilisation)))
    # nets: degree, pad, cluster
    d = np.arange(2, MAX_DEGREE + 1)
    p = d ** -synth.fit_powerlaw_alpha(MEAN_DEGREE, 2, MAX_DEGREE)
    deg = d[np.minimum(np.searchsorted(np.cumsum(p / p.sum()), rng.random(nn)), d.size - 1)]
    pad = rng.random(nn) < 0.05
    k_cells = np.maximum(np.minimum(deg, nc // 4) - pad, 1)
    root = rng.integers(0, nc, nn)
    root[:nc] = rng.permutation(nc)
    level = np.maximum(rng.geometric(1.0 - RENT_P, nn) - 1, np.ceil(np.log2(k_cells * 2.0 / LEAF)).clip(0).astype(np.int64))
    size = np.minimum(LEAF * 2 ** np.minimum(level, 30), 2 ** int(math.log2(nc))).astype(np.int64)
    start = np.minimum(root // size * size, nc - size)
    # distinct cells of the cluster: an odd stride over a power of two
    stride = 2 * rng.integers(0, 1 << 20, nn) + 1
    deg = k_cells + pad
    net_start = np.concatenate([[0], np.cumsum(deg)])
    net = np.repeat(np.arange(nn), deg)
    k = np.arange(net_start[-1]) - net_start[net]
    owner = start[net] + (root[net] - start[net] + k * stride[net]) % size[net]
    last = net_start[1:][pad] - 1
    hx, hy = _home(root[pad], nc)
    edge = np.argmin(np.stack([hy, 1 - hx, 1 - hy, hx]), axis=0)
    along = np.choose(edge, [hx, hy, 1 - hx, 1 - hy])
    pad_id = ((edge + along) / 4 * nt).astype(np.int64) + rng.integers(-2, 3, hx.size)
    owner[owner >= nc] = 0
    n_nodes = nc + macros
    owner[last] = n_nodes + pad_id % nt
    if macros:  # four nets of three pins for each macro
        m = np.repeat(np.arange(macros + nf), 4)
        m_owner = np.where(m < macros, nc + m, n_nodes + nt + m - macros)
        extra = np.stack([m_owner, rng.integers(0, nc // 2, m.size), nc // 2 + rng.integers(0, nc // 2, m.size)], 1)
        owner = np.concatenate([owner, extra.ravel()])
        net_start = np.concatenate([net_start, net_start[-1] + 3 * np.arange(1, m.size + 1)])
    # pads on a ring outside the core, fixed macros inside on whole units
    t = (np.arange(nt) + 0.5) / nt * 4.0
    e, f = np.floor(t).astype(int), t - np.floor(t)
    tx = np.choose(e, [f * side, np.full(nt, side + 1.0), (1 - f) * side, np.full(nt, -2.0)])
    ty = np.choose(e, [np.full(nt, -2.0), f * side, np.full(nt, side + 1.0), (1 - f) * side])
    fw, fh = mw[macros:], ms[macros:]
    tx = np.concatenate([tx, np.rint(rng.uniform(0.1, 0.8, nf) * (side - fw))])
    ty = np.concatenate([ty, np.rint(rng.uniform(0.1, 0.8, nf) * (side - fh))])
    tw, th = np.concatenate([np.ones(nt), fw]), np.concatenate([np.ones(nt), fh])
    node_w, node_h = np.concatenate([w, mw[:macros]]), np.concatenate([np.ones(nc), ms[:macros]])
    dx = (rng.random(owner.size) - 0.5) * np.concatenate([node_w, tw])[owner]
    dy = (rng.random(owner.size) - 0.5) * np.concatenate([node_h, th])[owner]
    on_pad = (owner >= n_nodes) & (owner < n_nodes + nt)
    dx[on_pad] = dy[on_pad] = 0.0
    f32 = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    i32 = lambda a: np.ascontiguousarray(a, np.int32)  # noqa: E731
    rows = int(side)
    centre = f32(np.full(n_nodes, side / 2))
    nl = synth.Netlist(
        name="case", node_w=f32(node_w), node_h=f32(node_h), node_cx=centre, node_cy=centre.copy(), term_llx=f32(tx),
        term_lly=f32(ty), term_w=f32(tw), term_h=f32(th), term_is_ni=np.zeros(nt + nf, np.uint8),
        net_start=i32(net_start), pin_owner=i32(owner), pin_dx=f32(dx), pin_dy=f32(dy),
        row_llx=f32(np.zeros(rows)), row_lly=f32(np.arange(rows)), row_urx=f32(np.full(rows, side)),
        row_h=f32(np.ones(rows)), row_site_w=f32(np.ones(rows)), target_density=1.0, bins=bins)
    hx, hy = _home(np.arange(nc), nc)
    return nl, np.concatenate([hx, rng.uniform(0.1, 0.9, macros)]), np.concatenate([hy, rng.uniform(0.1, 0.9, macros)])


def _spread(rng, nl, hx, hy, spread):
    """Node centres `spread` of the way from the core centre to their homes."""
    side = nl.core()[2]
    xy = []
    for h, s in ((hx, nl.node_w), (hy, nl.node_h)):
        c = side * (0.5 + spread * (h - 0.5)) + rng.normal(0.0, 0.02 * side, h.size)
        half = 0.5 * s.astype(np.float64) + 1e-3
        xy.append(np.clip(c, half, side - half).astype(np.float32))
    return xy


def _design(case, seed):
    rng = np.random.default_rng([seed, case["cells"]])
    if case["kind"] == "place" and case["cells"] == 100:
        nl = synth.smoke(1)
        side = nl.core()[2]
        cx, cy = rng.uniform(0.25 * side, 0.75 * side, (2, nl.num_nodes))
        return nl.with_positions(cx, cy), rng
    nl, hx, hy = _netlist(rng, case["cells"], case.get("macros", 0), case.get("bins", 0))
    return nl.with_positions(*_spread(rng, nl, hx, hy, case.get("spread", 0.6))), rng


def _params(nl, case):
    return placer.default_params(
        target_density=float(nl.target_density), bins_x=int(nl.bins), bins_y=int(nl.bins),
        precision=placer.PREC_FP64 if case.get("fp64") else placer.PREC_MIXED,
        step_rule=placer.STEP_BB if case.get("rule") == "bb" else placer.STEP_LIPSCHITZ,
        wl_model=placer.WL_LSE if case.get("lse") else placer.WL_WA,
        exp_mode=placer.EXP_EXACT if case.get("exact_exp") else placer.EXP_FAST)


def _pinned(n, fp64=False):
    return torch.empty((n, 2), dtype=torch.float64 if fp64 else torch.float32, pin_memory=torch.cuda.is_available())


def _read(engine, out):
    """The positions of every object into a pinned buffer."""
    n = out.shape[0]
    if out.dtype == torch.float64:
        rc = placer.load().ep_get_positions_f64(engine.h, placer.MGP, ctypes.cast(out.data_ptr(), _F64P), n)
        if rc:
            raise placer.EPError(rc, "ep_get_positions_f64")
    else:
        engine.get_positions_ptr(out.data_ptr(), n)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scatter":
        d = _scatter_inputs(case, seed)
        dev = {k: torch.from_numpy(v).cuda() for k, v in d["arrays"].items()}
        out = [torch.empty((case["bins"], case["bins"]), dtype=torch.float32, device="cuda") for _ in range(2)]
        g = d["grid"]
        return dict(case=case, grid=placer.ScatterGrid(g["bins"], g["bins"], 0.0, 0.0, g["step"], g["step"], 1.0),
                    dev=dev, out=out)
    if kind == "batch":
        sizes = np.random.default_rng([case["cells"], case["designs"]])
        sizes = np.exp(sizes.uniform(math.log(case["cells"]), math.log(case["top"]), case["designs"])).astype(int)
        nls = [_design(dict(kind=kind, cells=int(n)), seed * 64 + k)[0] for k, n in enumerate(sizes)]
        engines = placer.create_engines(nls, [_params(nl, case) for nl in nls])
        for e in engines:
            e.save_positions()
        return dict(case=case, engines=engines, out=[_pinned(e.info.num_objects) for e in engines])
    nl, rng = _design(case, seed)
    e = placer.Engine(nl, _params(nl, case))
    s = dict(case=case, engine=e, out=_pinned(e.info.num_objects, case.get("fp64") and kind == "place"))
    if kind == "gradient":
        # lambda_0 at one placement; the gradient is asked for at another
        e.set_positions(_gradient_positions(nl, rng, e.info.num_objects))
        e.initialize()
        s["xy"] = _pinned(e.info.num_objects)
        s["xy"].copy_(torch.from_numpy(_gradient_positions(nl, rng, e.info.num_objects)))
    elif kind in ("start", "train"):
        w, s["start"] = warmstart.load_weights()
        s["gnn"] = placer.Gnn(weights=w)
        if kind == "train":
            s["target"] = _targets(nl, rng)
    if kind in ("place", "qp", "start"):
        e.save_positions()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "scatter":
        d = s["dev"]
        rc, msg = placer.density_scatter_noalloc(s["grid"], d["cx"].numel(), d["cx"].data_ptr(), d["cy"].data_ptr(),
                                                 d["w"].data_ptr(), d["h"].data_ptr(), d["flags"].data_ptr(),
                                                 s["out"][0].data_ptr(), s["out"][1].data_ptr(),
                                                 torch.cuda.current_stream().cuda_stream)
        if rc:
            raise placer.EPError(rc, msg)
        return s["out"]
    if kind == "batch":
        for e in s["engines"]:
            e.load_positions()
            e.initialize()
        stats = placer.run_batch(s["engines"], case["steps"])
        return [_read(e, o) for e, o in zip(s["engines"], s["out"])] + [[st["iterations"] for st in stats]]
    e, out = s["engine"], s["out"]
    if kind == "place":
        e.load_positions()
        e.initialize()
        st = e.nesterov_run(case["steps"])
        return [_read(e, out), st["iterations"]]
    if kind == "gradient":
        e.set_positions_ptr(s["xy"].data_ptr(), out.shape[0])
        e.eval_gradient()
        rc = placer.load().ep_get_gradient(e.h, placer.MGP, ctypes.cast(out.data_ptr(), _F32P), out.shape[0])
        if rc:
            raise placer.EPError(rc, "ep_get_gradient")
        q = e.query()
        return [out, q["overflow"], q["hpwl"]]
    if kind == "qp":
        e.load_positions()
        st = e.quadratic_placement(case["rounds"] - 1)
        return [_read(e, out), st["rounds"]]
    if kind == "start":
        e.load_positions()
        s["gnn"].release(e)  # the graph and the features anew, as for a design not seen before
        warmstart.propose(s["gnn"], e, s["start"])
        return _read(e, out)
    s["gnn"].release(e)
    loss, grad = s["gnn"].loss_grad(e, s["target"])
    return [loss, grad]


# -------------------------------------------------- what a pass cannot do without --
def _sizes(cells, macros=0, bins=0):
    nodes = cells + macros
    pins = 3.6 * 1.1 * cells
    objects = 1.45 * nodes
    b = bins or 2 ** max(2, min(10, int(math.log2(math.sqrt(1.45 * cells)))))
    return nodes, pins, objects, b * b


def _step_work(case, cells=None):
    """One evaluation and step: positions, sizes, gradients and optimizer
    vectors of the objects, the pins, the bin maps, each once; four
    exponentials a pin, the overlaps, the transforms."""
    nodes, pins, objects, bins = _sizes(cells or case["cells"], case.get("macros", 0), case.get("bins", 0))
    q = 2 if case.get("fp64") else 1
    return (128 * q * objects + 40 * q * bins + 12 * pins + 4 * 1.1 * nodes + 16 * q * nodes,
            100 * pins + 150 * objects + 15 * bins * math.log2(bins))


def work(case):
    kind = case["kind"]
    if kind == "place":
        b, f = _step_work(case)
        return dict(bytes=(case["steps"] + 1) * b, flops=(case["steps"] + 1) * f)
    if kind == "gradient":
        b, f = _step_work(case)
        return dict(bytes=b, flops=f)
    if kind == "batch":
        mean = (case["top"] - case["cells"]) / math.log(case["top"] / case["cells"])
        b, f = _step_work(case, cells=int(mean))
        return dict(bytes=case["designs"] * (case["steps"] + 1) * b, flops=case["designs"] * (case["steps"] + 1) * f)
    if kind == "scatter":
        return dict(bytes=17 * case["cells"] + 8 * case["bins"] ** 2, flops=120 * case["cells"])
    nodes, pins, objects, _ = _sizes(case["cells"])
    # entries of both systems, about 2.4 a pin and axis; a BiCGSTAB iteration
    # takes the matrix twice and about ten vectors
    it = 2 * (8 * 4.8 * pins) + 10 * 8 * nodes
    if kind == "qp":
        return dict(bytes=case["rounds"] * (100 * it + 80 * pins), flops=case["rounds"] * 100 * (4 * 4.8 * pins + 40 * nodes))
    # diffusion: 128 steps over the pins both ways; network: features, three
    # layers of two aggregations and a 128 x 64 product
    diff = 128 * (8 * pins + 24 * nodes)
    fwd_b = 3 * (2 * 256 * nodes + 8 * pins + 2 * 256 * nodes) + 300 * nodes
    fwd_f = 3 * (2 * 2 * 64 * pins + 2 * 64 * 128 * nodes) + 2 * 64 * 13 * nodes
    if kind == "start":
        return dict(bytes=diff + fwd_b + 20 * it + 80 * pins, flops=128 * 4 * pins + fwd_f + 20 * 4 * 4.8 * pins)
    return dict(bytes=diff + 3 * fwd_b, flops=128 * 4 * pins + 3 * fwd_f)


# ------------------------------------------------ inputs and values in 64 bits --
def _scatter_inputs(case, seed):
    rng = np.random.default_rng([seed, case["cells"], case["bins"]])
    n = case["cells"]
    w = np.clip(np.rint(rng.lognormal(math.log(3.0) - 0.18, 0.6, n)), 1, 20)
    h = np.ones(n)
    flags = (rng.random(n) < 0.3).astype(np.uint8) * np.uint8(FILLER)
    big = rng.random(n) < 2e-5
    w[big], h[big], flags[big] = rng.integers(8, 60, big.sum()), rng.integers(8, 60, big.sum()), MACRO
    side = math.ceil(math.sqrt((w * h).sum()))
    hx, hy = _home(np.arange(n), n)
    a = dict(w=w, h=h)
    for k, home, s in (("cx", hx, w), ("cy", hy, h)):
        c = side * (0.5 + case["spread"] * (home - 0.5)) + rng.normal(0.0, 0.02 * side, n)
        half = np.maximum(0.5 * s, 0.5 * side / case["bins"]) + 1e-2
        a[k] = np.clip(c, half, side - half)
    a = {k: np.ascontiguousarray(v, np.float32) for k, v in a.items()}
    return dict(arrays=dict(a, flags=flags), grid=dict(bins=case["bins"], step=float(np.float32(side / case["bins"]))))


def _targets(nl, rng):
    """Quadratic placement and final centres of a design: its cells pulled
    half-way to the centre, and at their homes."""
    side = nl.core()[2]
    hx, hy = _home(np.arange(nl.num_nodes), nl.num_nodes)
    home = np.stack([hx, hy], 1)
    q = 0.5 + 0.5 * (home - 0.5) + rng.normal(0, 0.02, home.shape)
    f = home + rng.normal(0, 0.02, home.shape)
    return np.ascontiguousarray(side * np.clip(np.concatenate([q, f], 1), 0.01, 0.99), np.float32)


def _gradient_positions(nl, rng, objects):
    """Where the gradient is asked for: the nodes moved a little from the
    start, the fillers anywhere in the core."""
    side, n = nl.core()[2], nl.num_nodes
    xy = rng.uniform(0.02 * side, 0.98 * side, (objects, 2))
    for c, (p, s) in enumerate(((nl.node_cx, nl.node_w), (nl.node_cy, nl.node_h))):
        half = 0.5 * s.astype(np.float64) + 1e-3
        xy[:n, c] = np.clip(p + rng.normal(0, 0.005 * side, n), half, side - half)
    return np.ascontiguousarray(xy, np.float32)


def _spans(lo, hi, step, bins):
    i0 = np.maximum((lo / step).astype(np.int64), 0)
    return i0, np.minimum((hi / step).astype(np.int64), bins - 1)


def _rects(c, size, step):
    """Low and high edges and the smoothing scale along one axis."""
    half = 0.5 * np.where(size < step, step, size)
    return c - half, c + half, np.where(size < step, size / step, 1.0)


def _overlaps(cx, cy, w, h, step, bins):
    """(object, bin x, bin y, overlap area times smoothing) of every pair."""
    lx, hx, sx = _rects(cx, w, step[0])
    ly, hy, sy = _rects(cy, h, step[1])
    i0, i1 = _spans(lx, hx, step[0], bins)
    j0, j1 = _spans(ly, hy, step[1], bins)
    nx, ny = np.maximum(i1 - i0 + 1, 0), np.maximum(j1 - j0 + 1, 0)
    o = np.repeat(np.arange(cx.size), nx * ny)
    k = np.arange(o.size) - np.repeat(np.cumsum(nx * ny) - nx * ny, nx * ny)
    i, j = i0[o] + k // ny[o], j0[o] + k % ny[o]
    ox = np.minimum(hx[o], (i + 1) * step[0]) - np.maximum(lx[o], i * step[0])
    oy = np.minimum(hy[o], (j + 1) * step[1]) - np.maximum(ly[o], j * step[1])
    return o, i, j, np.maximum(ox, 0) * np.maximum(oy, 0) * (sx * sy)[o]


def _poisson(rho, step):
    nx, ny = rho.shape
    wx, wy = np.pi * np.arange(nx) / nx, np.pi * np.arange(ny) / ny * (step[1] / step[0])
    ax = np.outer(np.arange(nx), np.arange(nx) + 0.5) * np.pi / nx
    ay = np.outer(np.arange(ny), np.arange(ny) + 0.5) * np.pi / ny
    half = np.outer(np.where(np.arange(nx), 1, 0.5), np.where(np.arange(ny), 1, 0.5))
    den = wx[:, None] ** 2 + wy[None, :] ** 2
    den[0, 0] = 1.0
    k = 4.0 / nx / ny * half / den
    k[0, 0] = 0.0
    p = np.cos(ax) @ rho @ np.cos(ay).T * k
    return np.sin(ax).T @ (wx[:, None] * p) @ np.cos(ay), np.cos(ax).T @ (p * wy[None, :]) @ np.sin(ay)


def _wirelength(x, start, net, inv_gamma, lse, exact_exp):
    """Gradient at every pin along one axis."""
    hi, lo = np.maximum.reduceat(x, start), np.minimum.reduceat(x, start)
    g = np.zeros(x.size)
    for sign, ext in ((1.0, hi), (-1.0, lo)):
        a = sign * (x - ext[net]) * inv_gamma
        e = np.where(a > -300.0, np.exp(a) if exact_exp else (1.0 + a / 1024.0) ** 1024, 0.0)
        share = e / np.add.reduceat(e, start)[net]
        if not lse:
            share = share * (1.0 + sign * (x - np.add.reduceat(share * x, start)[net]) * inv_gamma)
        g += sign * share
    return g


def _evaluate(nl, case, xy, fillers, filler_size, lam, bins):
    """(direction, overflow, HPWL, sum |wirelength gradient|, sum |density
    gradient|) at centres xy of the nodes and the fillers."""
    n, side = nl.num_nodes, float(nl.core()[2])
    f8 = lambda a: np.asarray(a, np.float64)  # noqa: E731
    w = np.concatenate([f8(nl.node_w), np.full(fillers, filler_size[0])])
    h = np.concatenate([f8(nl.node_h), np.full(fillers, filler_size[1])])
    step = (float(np.float32(side) / np.float32(bins)),) * 2
    bin_area = step[0] * step[1]
    o, i, j, a = _overlaps(xy[:, 0], xy[:, 1], w, h, step, bins)
    flat = i * bins + j
    node = np.bincount(flat[o < n], a[o < n], bins * bins)
    fill = np.bincount(flat[o >= n], a[o >= n], bins * bins)
    term = np.zeros(bins * bins)
    inside = (nl.term_llx >= 0) & (nl.term_lly >= 0) & (nl.term_llx + nl.term_w <= side) & (nl.term_lly + nl.term_h <= side)
    for t in np.nonzero(inside)[0]:
        lo = f8([nl.term_llx[t], nl.term_lly[t]])
        hi = lo + f8([nl.term_w[t], nl.term_h[t]])
        e = np.arange(bins) * step[0]
        ox, oy = (np.maximum(np.minimum(hi[c], e + step[0]) - np.maximum(lo[c], e), 0) for c in range(2))
        term += np.outer(ox, oy).ravel()
    area = f8(nl.node_w) * f8(nl.node_h)
    over = np.maximum((node + term) / bin_area - 1.0, 0.0).sum() * bin_area / area.sum()
    ex, ey = _poisson(((node + fill + term) / bin_area).reshape(bins, bins), step)
    gd = np.stack([np.bincount(o, a * e[i, j], n + fillers) for e in (ex, ey)], 1)
    t = 0.1 if over > 1.0 else 10.0 if over < 0.1 else 1.0 / 10.0 ** ((over - 0.1) * 20 / 9.0 - 1.0)
    inv_gamma = 0.125 / step[0] * t
    start, owner = nl.net_start[:-1].astype(np.int64), nl.pin_owner
    net = np.repeat(np.arange(nl.num_nets), np.diff(nl.net_start))
    centres = np.concatenate([xy[:n], np.stack([f8(nl.term_llx) + 0.5 * f8(nl.term_w), f8(nl.term_lly) + 0.5 * f8(nl.term_h)], 1)])
    gw, hpwl = np.zeros((n + fillers, 2)), 0.0
    for c, off in enumerate((nl.pin_dx, nl.pin_dy)):
        x = centres[owner, c] + f8(off)
        hpwl += (np.maximum.reduceat(x, start) - np.minimum.reduceat(x, start)).sum()
        g = _wirelength(x, start, net, inv_gamma, case.get("lse"), case.get("exact_exp"))
        gw[:n, c] = np.bincount(owner, g, n + nl.num_terminals)[:n]
    pins = np.concatenate([np.bincount(owner, minlength=n)[:n], np.zeros(fillers)])
    pre = 1.0 / np.maximum(1.0, pins + lam * w * h)
    return pre[:, None] * (lam * gd - gw), over, hpwl, np.abs(gw).sum(), np.abs(gd).sum()


def _fillers(nl):
    """Number and size of the fillers of a design whose areas are whole
    numbers, and the bins a side that the automatic rule gives."""
    side = float(nl.core()[2])
    area = np.sort(nl.node_w.astype(np.float64) * nl.node_h)
    inside = nl.term_llx >= 0
    inside &= (nl.term_lly >= 0) & (nl.term_llx < side) & (nl.term_lly < side)
    fixed = (nl.term_w[inside].astype(np.float64) * nl.term_h[inside]).sum()
    n = area.size
    lo, hi = int(0.05 * np.float32(n)), int(0.95 * np.float32(n))
    each = np.float32(area[lo:hi].sum()) / np.float32(hi - lo)
    count = max(0, int(np.float32(np.float32(side * side - fixed - area.sum()) / each) + 0.5))
    ideal = int(np.float32(side * side) / (np.float32(area.sum()) / np.float32(n)) + np.float32(0.5))
    bins = next((2 << i for i in range(1, 10) if (2 << i) ** 2 <= ideal < (4 << i) ** 2), 1024)
    return count, (float(each), 1.0), nl.bins or bins


def _exact_gradient(case, seed):
    nl, rng = _design(case, seed)
    count, size, bins = _fillers(nl)
    first, xy = (_gradient_positions(nl, rng, nl.num_nodes + count).astype(np.float64) for _ in range(2))
    w, d = _evaluate(nl, case, first, count, size, 0.0, bins)[3:]
    return list(_evaluate(nl, case, xy, count, size, float(np.float32(w / d)), bins)[:3])


def _exact_train(case, seed):
    nl, rng = _design(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    n, nt, side = nl.num_nodes, nl.num_terminals, float(nl.core()[2])
    net = torch.as_tensor(np.repeat(np.arange(nl.num_nets), np.diff(nl.net_start)), device=dev)
    node = torch.as_tensor(nl.pin_owner.astype(np.int64), device=dev)
    deg = T(np.diff(nl.net_start))[:, None]
    pins = torch.zeros(n + nt, dtype=torch.float64, device=dev).index_add_(0, node, torch.ones_like(node, dtype=torch.float64))
    movable = (node < n).to(torch.float64)[:, None]

    def aggregate(v):
        a = torch.zeros(nl.num_nets, v.shape[1], dtype=v.dtype, device=dev).index_add(0, net, v[node]) / deg
        return torch.zeros_like(v).index_add(0, node, a[net] * movable) / pins.clamp(min=1.0)[:, None]

    x = torch.zeros(n + nt, 9, dtype=torch.float64, device=dev)
    x[:n, 0] = torch.log1p(T(nl.node_w) * T(nl.node_h)) * 0.25
    x[:, 1] = torch.log1p(pins) / 3.0
    x[n:, 2] = 1.0
    pads = torch.stack([T(nl.term_llx) + 0.5 * T(nl.term_w), T(nl.term_lly) + 0.5 * T(nl.term_h)], 1) / side
    v = torch.cat([torch.full((n, 2), 0.5, dtype=torch.float64, device=dev), pads])
    on_net = (pins[:n] > 0)[:, None]
    for k in range(1, 129):
        v = torch.cat([torch.where(on_net, aggregate(v)[:n], v[:n]), pads])
        if k in (8, 32, 128):
            x[:, 3 + 2 * (8, 32, 128).index(k):][:, :2] = v
    w = torch.as_tensor(warmstart.load_weights()[0], device=dev)
    parts, at = [], 0
    for rows, cols in [(64, 9), (64, 1)] + 3 * [(64, 128), (64, 1)] + [(4, 64), (4, 1)]:
        p = w[at:at + rows * cols].reshape(rows, cols)
        # the forward pass takes the weights in BF16, the biases in FP32
        parts.append((p.to(torch.bfloat16) if cols > 1 else p).to(torch.float64).requires_grad_(True))
        at += rows * cols
    h = torch.relu(x @ parts[0].T + parts[1].T)
    for l in (2, 4, 6):
        h = torch.relu(torch.cat([h, aggregate(h)], 1) @ parts[l].T + parts[l + 1].T)
    raw = h @ parts[8].T + parts[9].T
    pred = torch.cat([v, v], 1) + 0.25 * torch.tanh(raw)
    loss = ((pred[:n] - T(_targets(nl, rng)) / side) ** 2).sum() / (2 * n)
    loss.backward()
    return [loss.item(), torch.cat([p.grad.reshape(-1) for p in parts])]


def exact(case, seed):
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "scatter":
        d = _scatter_inputs(case, seed)
        a, g = {k: v.astype(np.float64) for k, v in d["arrays"].items()}, d["grid"]
        o, i, j, area = _overlaps(a["cx"], a["cy"], a["w"], a["h"], (g["step"], g["step"]), g["bins"])
        filler = (d["arrays"]["flags"] & FILLER) != 0
        return [np.bincount((i * g["bins"] + j)[m], area[m], g["bins"] ** 2).reshape(g["bins"], -1)
                for m in (~filler[o], filler[o])]
    return None  # an iteration from a start: no closed value
