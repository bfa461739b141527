"""The fast-transform Poisson solve at the sizes where its passes differ: 2,
3 or 4 stages in the first pass over a sequence (log2 n mod 3), one pass or
several.  In FP64: the same templates run in FP32 at square sizes against the
same oracle elsewhere; on very oblong grids FP32's own rounding, not the
passes, decides the field across the short side.

Tolerance: 2e-6 of max|E| (max|phi|) of the FP64 dense restatement on the
engine's own density map, as for the square sizes: the maps are read in FP32."""
import numpy as np
import pytest

from eplace_b200 import placer, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bx,by", [(8, 2048), (16, 16), (32, 1024), (64, 512), (128, 32), (1024, 8), (2048, 1024)])
def test_field_at_each_pass_split(bx, by):
    nl = synth.blob_start(synth.standard_cell(4_000, seed=9), sigma_frac=0.2)
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=bx, bins_y=by, precision=placer.PREC_FP64,
                                                dct_mode=placer.DCT_FFT, keep_maps=1))
    e.initialize()
    m = e.bin_maps()
    i = e.info
    bin_area = np.float64(np.float32(i.bin_step_x) * np.float32(i.bin_step_y))
    rho = (m["node"].astype(np.float64) + m["base"] + m["filler"] + m["terminal"]) / bin_area
    ex, ey, phi = O.poisson(rho, i.bin_step_x, i.bin_step_y)
    scale = max(np.abs(ex).max(), np.abs(ey).max())
    assert max(np.abs(m["ex"] - ex).max(), np.abs(m["ey"] - ey).max()) < 2e-6 * scale
    assert np.abs(m["phi"] - phi).max() < 2e-6 * np.abs(phi).max()
    e.close()
