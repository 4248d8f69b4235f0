"""The FP32 expansion beyond the sizes where a centre gets a block of its own:
16 copies of a box (1 920 centres) with many and with few neighbours, and one
box (120 centres) at chunks of 32, 64 and 128 pairs.

Tolerance: the FP32 features' bar, 1e-5 of the largest value."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import tune
from oracle import oracle as O
from test_gpu_nl_sorts import grid_box
from test_gpu_parity import oracle_calc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,l", [(1, 0), (3, 2), (8, 6), (11, 9), (16, 12)])
@pytest.mark.parametrize("copies,side,chunk", [(16, 6.0, None), (16, 14.0, None), (1, 6.0, 8), (1, 6.0, 16), (1, 6.0, 32)])
def test_features(n, l, copies, side, chunk):
    batch = grid_box(120, side, n + l, species=(8, 14))
    batch["numbers"][5] = 1
    species = [1, 8, 14]
    calc = rb.SphericalExpansion(interaction_cutoff=4.0, cutoff_smooth_width=0.5, max_radial=n, max_angular=l,
                                 gaussian_sigma_type="Constant", gaussian_sigma_constant=0.5)
    many = dict(atom_offsets=np.arange(copies + 1) * 120, positions=np.concatenate([batch["positions"]] * copies),
                numbers=np.concatenate([batch["numbers"]] * copies), cells=np.concatenate([batch["cells"]] * copies),
                pbc=np.concatenate([batch["pbc"]] * copies))
    before = tune.get_config((3, n, l)) if chunk else None
    if chunk:
        tune.set_config((3, n, l), dict(before, exp_chunk=chunk))
    try:
        al = calc.transform(rb.AtomsList(rb.StructureSet(many)), precision="fp32")
        c = al.get_features(calc, keys=calc.get_keys(species)).reshape(copies, 120, -1)
    finally:
        if chunk:
            tune.set_config((3, n, l), before)
    ref = O.Run(oracle_calc(rc=4.0, n=n, l=l, sigma=0.5), batch, species).expansion().reshape(c.shape[1:])
    assert np.abs(c - ref).max() <= 1e-5 * np.abs(ref).max()
