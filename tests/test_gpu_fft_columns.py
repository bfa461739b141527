"""The FP32 fast-transform Poisson solve where it differs from the FP64 one: four
columns to a block from 1024 bins in y on, on square and oblong grids, and 2048
bins on either axis.  The reference is the factorization in float64, itself
checked against the dense oracle on the CPU.

Tolerance: twice the 2e-6 of max|E| (max|phi|) that the sizes up to 1024^2 are
held to: a transform of 2048 adds one stage of eleven to the roundings, and the
maps here are sparser (five times the bins a cell), so their peak field is
smaller against the sums that are rounded."""
import numpy as np
import pytest

from eplace_b200 import placer, synth
from tests.test_fft_factorization import fft_poisson

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bx,by", [(256, 1024), (512, 1024), (2048, 1024), (512, 2048), (1024, 2048), (2048, 2048),
                                   (2048, 512)])
def test_fp32_field_of_the_large_grids(bx, by):
    nl = synth.blob_start(synth.standard_cell(20_000, seed=5), sigma_frac=0.15)
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=bx, bins_y=by, dct_mode=placer.DCT_FFT,
                                                keep_maps=1))
    e.initialize()
    m, i = e.bin_maps(), e.info
    bin_area = np.float64(np.float32(i.bin_step_x) * np.float32(i.bin_step_y))
    rho = (m["node"].astype(np.float64) + m["base"] + m["filler"] + m["terminal"]) / bin_area
    ex, ey, phi = fft_poisson(rho, float(i.bin_step_x), float(i.bin_step_y))
    scale = max(np.abs(ex).max(), np.abs(ey).max())
    assert max(np.abs(m["ex"] - ex).max(), np.abs(m["ey"] - ey).max()) < 4e-6 * scale
    assert np.abs(m["phi"] - phi).max() < 4e-6 * np.abs(phi).max()
    e.close()
