"""The per-net pass by net degree: each form's first and last degree (a thread
per net, a lane per pin, a warp per net, a block per net and its chunks)
against the FP64 oracle, on geometry whose pin positions are exact in float."""
import numpy as np
import pytest

from eplace_b200 import placer, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def degree_design(degrees, nets_each, seed):
    """Nets of the given degrees in a seeded order, every pin on a cell of its
    own but for one in eight, which shares a cell, and one pin in 50 on a pad."""
    rng = np.random.default_rng(seed)
    deg = rng.permutation(np.repeat(degrees, nets_each))
    pins = int(deg.sum())
    n, nt, side = max(64, pins - pins // 8), 4, 128.0
    owner = rng.permutation(np.concatenate([np.arange(n), rng.integers(0, n, max(0, pins - n))]))[:pins]
    owner[rng.random(pins) < 0.02] = n + rng.integers(0, nt)
    f = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    q = lambda lo, hi, k: np.round(rng.uniform(lo, hi, k) * 16) / 16  # noqa: E731
    rows = int(side)
    return synth.Netlist(
        name="degrees", node_w=f(np.ones(n)), node_h=f(np.ones(n)), node_cx=f(q(2, side - 2, n)),
        node_cy=f(q(2, side - 2, n)), term_llx=f([-2, side + 1, 10, 20]), term_lly=f([10, 20, -2, side + 1]),
        term_w=f(np.ones(nt)), term_h=f(np.ones(nt)), term_is_ni=np.ones(nt, np.uint8),
        net_start=np.concatenate([[0], np.cumsum(deg)]).astype(np.int32), pin_owner=owner.astype(np.int32),
        pin_dx=f(q(-0.5, 0.5, pins)), pin_dy=f(q(-0.5, 0.5, pins)), row_llx=f(np.zeros(rows)),
        row_lly=f(np.arange(rows)), row_urx=f(np.full(rows, side)), row_h=f(np.ones(rows)),
        row_site_w=f(np.ones(rows)), bins=32)


# nets of one degree in counts that fill a warp's or a block's task and spill
# by one; 128 and 256 pins are a chunk of the block form in FP64 and FP32
DEGREES = [(1, 33), (2, 33), (3, 64), (4, 257), (5, 31), (6, 6), (7, 5), (8, 4), (16, 3), (17, 2), (31, 2), (32, 2),
           (33, 2), (96, 3), (97, 2), (128, 1), (129, 1), (256, 1), (257, 1), (600, 2)]


@pytest.mark.parametrize("lse", [False, True])
@pytest.mark.parametrize("precision", [placer.PREC_MIXED, placer.PREC_FP64])
@pytest.mark.parametrize("degrees", [[d] for d in DEGREES] + [DEGREES], ids=lambda d: "all" if len(d) > 1 else str(d[0][0]))
def test_gradient_and_hpwl_by_degree(degrees, precision, lse):
    nl = degree_design([d for d, _ in degrees], [k for _, k in degrees], seed=len(degrees) + degrees[0][0])
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=32, bins_y=32, precision=precision, keep_maps=1,
                                                wl_model=placer.WL_LSE if lse else placer.WL_WA))
    e.eval_gradient()
    s = e.query()
    xy = e.get_positions().astype(np.float64)
    gw = e.component_gradients_f64()[1]
    n, nf = nl.num_nodes, e.info.num_fillers
    obj = nl.with_positions(nl.node_cx, nl.node_cy)
    obj.pin_owner = np.where(nl.pin_owner >= n, nl.pin_owner + nf, nl.pin_owner).astype(np.int32)
    _, hp, ref = O.wirelength_grad(obj, xy[:, 0], xy[:, 1], nl.term_llx + 0.5, nl.term_lly + 0.5, s["inv_gamma_x"],
                                   s["inv_gamma_y"], lse=lse)
    # fastExp is ten squarings of 1 + a / 1024: 2047 roundings of 2^-24 in FP32
    # (1.2e-4) in each of two terms and their sums; of 2^-53 (2.3e-13) in FP64
    tol = 5e-4 if precision == placer.PREC_MIXED else 1e-9
    assert np.abs(gw[:n] - ref[:n]).max() <= tol * max(np.abs(ref[:n]).max(), 1.0)
    # the bound pins are exact here, so only the order of the FP64 sum differs
    assert s["hpwl"] == pytest.approx(hp, rel=1e-12)
    assert e.hpwl() == s["hpwl"]
    e.close()
