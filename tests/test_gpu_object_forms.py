"""Scatter, gather and direction by object footprint: a thread per object with
one, two and more rows of bins, a warp and a block per kBig object, and lanes
paired for the atomics, against the FP64 oracle on geometry exact in float."""
import numpy as np
import pytest

from eplace_b200 import placer, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIDE, BINS = 128.0, 64  # bins of 2 x 2
# small objects within one, two and three rows of bins (at most 16 bins), the
# first footprint of a warp, a wide and a square warp object, and blocks
SIZES = {
    "cells": [(1, 1), (2, 1), (3, 1), (5, 1), (11, 1)],
    "rows": [(1, 2), (2, 3), (3, 4), (1, 9), (2, 11)],
    "warp": [(13, 1), (30, 1), (6, 6), (40, 20), (1, 60)],
    "block": [(48, 38), (64, 40), (3, 127), (127, 24)],
}
SIZES["all"] = [s for k in ("cells", "rows", "warp", "block") for s in SIZES[k]]


def sized_design(sizes, count, seed):
    rng = np.random.default_rng(seed)
    wh = np.array([sizes[k % len(sizes)] for k in range(count)], np.float64)
    wh = np.concatenate([wh, np.ones((35, 2))])  # a last warp that is not full
    n, nt, rows = len(wh), 4, int(SIDE)
    # centres on sixteenths, the objects inside the core
    half = wh / 2
    c = np.round((half + rng.random((n, 2)) * (SIDE - wh)) * 16) / 16
    c = np.clip(c, half, SIDE - half)
    owner = np.concatenate([rng.permutation(n), rng.integers(0, n, n)])
    deg = np.full(len(owner) // 2, 2)
    f = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    return synth.Netlist(
        name="sizes", node_w=f(wh[:, 0]), node_h=f(wh[:, 1]), node_cx=f(c[:, 0]), node_cy=f(c[:, 1]),
        term_llx=f([-2, SIDE + 1, 10, 20]), term_lly=f([10, 20, -2, SIDE + 1]), term_w=f(np.ones(nt)), term_h=f(np.ones(nt)),
        term_is_ni=np.ones(nt, np.uint8), net_start=np.concatenate([[0], np.cumsum(deg)]).astype(np.int32),
        pin_owner=owner[:deg.sum()].astype(np.int32), pin_dx=f(np.zeros(deg.sum())), pin_dy=f(np.zeros(deg.sum())),
        row_llx=f(np.zeros(rows)), row_lly=f(np.arange(rows)), row_urx=f(np.full(rows, SIDE)), row_h=f(np.ones(rows)),
        row_site_w=f(np.ones(rows)), bins=BINS)


@pytest.mark.parametrize("precision", [placer.PREC_MIXED, placer.PREC_FP64])
@pytest.mark.parametrize("kind,count", [("cells", 1500), ("rows", 700), ("warp", 60), ("block", 4), ("all", 40)])
def test_density_and_gather_by_footprint(kind, count, precision):
    nl = sized_design(SIZES[kind], count, seed=count)
    fp64 = precision == placer.PREC_FP64
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=BINS, bins_y=BINS, precision=precision, keep_maps=1))
    i = e.info
    assert i.bin_step_x == 2.0 and i.bin_step_y == 2.0
    e.set_positions(np.round(e.get_positions() * 16) / 16)
    e.eval_gradient()
    xy, n, nf = e.get_positions().astype(np.float64), nl.num_nodes, i.num_fillers
    w = np.concatenate([nl.node_w, np.full(nf, i.filler_w, np.float32)])
    h = np.concatenate([nl.node_h, np.full(nf, i.filler_h, np.float32)])
    flags = np.concatenate([(nl.node_h > 1).astype(np.uint8) * O.MACRO, np.full(nf, O.FILLER, np.uint8)])
    g = O.make_grid(BINS, BINS, (0.0, 0.0, SIDE, SIDE), 2.0, 2.0, 1.0)
    nd, fd, nq, fq = O.scatter(g, xy[:, 0], xy[:, 1], w, h, flags, i.density_scale)
    node_q, filler_q = e.density_fixed()
    assert np.array_equal(node_q, nq)  # node sizes and centres are exact, so both precisions agree
    if not fp64:
        assert np.array_equal(filler_q, fq)
    f = e.field_f64()
    gd = e.component_gradients_f64()[0]
    ref = O.gather(g, xy[:, 0], xy[:, 1], w, h, f["ex"], f["ey"])
    size = O.gather(g, xy[:, 0], xy[:, 1], w, h, np.abs(f["ex"]), np.abs(f["ey"]))
    # the nodes' overlaps are exact; a sum of at most 3000 products in partial
    # sums of at most 24 and trees: under 64 roundings of each term
    tol = 64 * (2.0 ** -53 if fp64 else 2.0 ** -24)
    assert (np.abs(gd[:n] - ref[:n]) <= tol * size[:n] + 1e-30).all()
    # the fused update scatters what it moved: a loop on its maps (keep_maps 0)
    # takes the same steps as one that scatters each evaluation anew
    b = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=BINS, bins_y=BINS, precision=precision, keep_maps=0))
    b.set_positions(xy)
    b.initialize()
    b.nesterov_run(3)
    c = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=BINS, bins_y=BINS, precision=precision, keep_maps=1))
    c.set_positions(xy)
    c.initialize()
    c.nesterov_run(3)
    assert np.array_equal(b.get_positions_f64(), c.get_positions_f64())
    for x in (e, b, c):
        x.close()
