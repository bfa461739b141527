"""The quadratic solver at its limits: what its matrices may hold, the memory it
takes for them, and the restart when r0.r vanishes."""
import numpy as np
import pytest

from eplace_b200 import placer, synth
from tests.test_gpu_qp_layout import star_design

pytestmark = pytest.mark.gpu


# rows of windows where most places are padding: few long nets whose bound pins
# differ between the axes, many rows just under and over 32 entries
@pytest.mark.parametrize("n,degrees", [
    (768, [33] * 135), (112, [80] * 39), (158, [80] * 34), (256, [17] * 400), (257, [33] * 9 + [2] * 40),
    (300, [32] * 300), (513, [9] * 500 + [33] * 16), (600, [5] * 2500),
], ids=lambda v: str(v) if isinstance(v, int) else "")
def test_matrix_fits_what_is_allocated(n, degrees):
    nl = star_design(n, degrees, seed=n)
    # hubs: the first eighth of the cells far out in x, the second in y
    k = n // 8
    nl.node_cx[:k] += 40
    nl.node_cy[k:2 * k] += 40
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=32, bins_y=32))
    e.quadratic_refine(1, 20)  # an overflow is EP_ERR_STATE
    assert e.quadratic_placement(3)["rounds"] == 4
    e.close()


def test_memory_follows_the_entries():
    """64 bytes a pin hold both matrices in full (four entries a pin and axis);
    the vectors and the layout take under 200 a cell.  Memory comes in chunks
    that double."""
    import torch
    nl = synth.standard_cell(20_000, seed=7, every_cell_pinned=True, local_pads=True)
    e = placer.Engine(nl, placer.default_params(target_density=1.0))
    free = torch.cuda.mem_get_info()[0]
    e.quadratic_placement(1)
    used = free - torch.cuda.mem_get_info()[0]
    assert used <= 3 * (64 * nl.pin_owner.size + 200 * nl.num_nodes), used
    e.close()


def far_design(n):
    """Cells far from pads at x = 0 but for one at 1e-5, a net each: the solution
    is so small beside the start that r0.r vanishes before |r| is down to eps
    |b|."""
    rng = np.random.default_rng(1)
    f = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    tx, rows = np.zeros(n), 1200
    tx[0] = 1e-5
    return synth.Netlist(
        name="far", node_w=f(np.ones(n)), node_h=f(np.ones(n)), node_cx=f(rng.uniform(300, 500, n)),
        node_cy=f(rng.uniform(-400, 400, n)), term_llx=f(tx - 0.5), term_lly=f(rng.uniform(-300, 300, n)),
        term_w=f(np.ones(n)), term_h=f(np.ones(n)), term_is_ni=np.ones(n, np.uint8),
        net_start=(2 * np.arange(n + 1)).astype(np.int32),
        pin_owner=np.stack([np.arange(n), n + np.arange(n)], 1).ravel().astype(np.int32), pin_dx=f(np.zeros(2 * n)),
        pin_dy=f(np.zeros(2 * n)), row_llx=f(np.full(rows, -600)), row_lly=f(np.arange(rows) - 600.0),
        row_urx=f(np.full(rows, 600)), row_h=f(np.ones(rows)), row_site_w=f(np.ones(rows)), bins=32)


# preconditioned, the restart is owed after the first iteration, also where that
# is one of the last allowed; plain, somewhere inside the second or third chunk
@pytest.mark.parametrize("n,iterations,jacobi", [(7, 2, True), (7, 100, True), (33, 3, True), (257, 11, True),
                                                 (1001, 100, True), (33, 100, False), (257, 100, False)])
def test_restart_when_the_residual_turns_orthogonal(n, iterations, jacobi):
    nl = far_design(n)
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=32, bins_y=32))
    st = e.quadratic_refine(1, iterations, jacobi)
    # bounds (2), matrix (3), set-up (3, 4 with the preconditioner), the solution
    # stored, five kernels an iteration, and one a restart
    assert (st["kernel_launches"] - 9 - jacobi) % 5 == 1
    assert st["solver_iterations"] <= iterations
    xy = e.get_positions()[:n].astype(np.float64)
    # eps |b| over the weights, which differ by 800 / 25 at most: 4e-11; without
    # the restart the first iteration's rounding stays, 500 x 2^-24 = 3e-5
    assert np.abs(xy[1:, 0]).max() < 1e-10
    assert abs(xy[0, 0] - (np.float64(nl.term_llx[0]) + 0.5)) < 1e-10
    e.close()


def test_no_restart_past_the_last_iteration():
    e = placer.Engine(far_design(33), placer.default_params(target_density=1.0, bins_x=32, bins_y=32))
    st = e.quadratic_refine(1, 1, True)
    assert st["solver_iterations"] == 1 and (st["kernel_launches"] - 10) % 5 == 0
    e.close()
