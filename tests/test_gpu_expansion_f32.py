"""The FP32 expansion with many neighbours (species-sorted sums in registers):
more neighbours than its window of 96 pairs, a species without neighbours, each
register variant (n up to 8, 12 and 16), each number of lanes per pair in the
harmonics, and few neighbours beside it.

Tolerance: the FP32 features' bar, 1e-5 of the largest value."""
import numpy as np
import pytest

import librascal_b200 as rb
from oracle import oracle as O
from test_gpu_nl_sorts import grid_box
from test_gpu_parity import oracle_calc, soap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,l", [(1, 0), (4, 1), (7, 2), (8, 3), (9, 5), (12, 7), (13, 9), (16, 12)])
@pytest.mark.parametrize("side", [6.0, 8.5, 14.0])
def test_features(n, l, side):
    # about 145, 51 and 11 neighbours per centre
    batch = grid_box(120, side, n + l, species=(8, 14))
    batch["numbers"][5] = 1  # a species that few centres see
    kw = dict(rc=4.0, n=n, l=l, sigma=0.5)
    species = [1, 8, 14]
    calc = rb.SphericalExpansion(interaction_cutoff=4.0, cutoff_smooth_width=0.5, max_radial=n, max_angular=l,
                                 gaussian_sigma_type="Constant", gaussian_sigma_constant=0.5)
    al = calc.transform(rb.AtomsList(rb.StructureSet(batch)), precision="fp32")
    c = al.get_features(calc, keys=calc.get_keys(species))
    ref = O.Run(oracle_calc(**kw), batch, species).expansion().reshape(c.shape)
    assert np.abs(c - ref).max() <= 1e-5 * np.abs(ref).max()
