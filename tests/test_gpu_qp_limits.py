"""The quadratic solver at its limits: what its matrices may hold and the memory
it takes for them."""
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
