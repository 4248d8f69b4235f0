"""The FP32 expansion for few neighbours at the numbers of radial channels
n (l + 1) where a lane takes another one: around 32, 64, 96, 128 and the most
there are (208), at each number of pairs per chunk; 16 copies of a box (1 920
centres, more than get a block each) with about 11 and 51 neighbours.

Tolerance: the FP32 features' bar, 1e-5 of the largest value."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import tune
from oracle import oracle as O
from test_gpu_nl_sorts import grid_box
from test_gpu_parity import oracle_calc

pytestmark = pytest.mark.gpu


def copies_match_oracle(n, l, species, side, chunk=16, copies=16):
    batch = grid_box(120, side, n + l, species=species)
    calc = rb.SphericalExpansion(interaction_cutoff=4.0, cutoff_smooth_width=0.5, max_radial=n, max_angular=l,
                                 gaussian_sigma_type="Constant", gaussian_sigma_constant=0.5)
    many = dict(atom_offsets=np.arange(copies + 1) * 120, positions=np.concatenate([batch["positions"]] * copies),
                numbers=np.concatenate([batch["numbers"]] * copies), cells=np.concatenate([batch["cells"]] * copies),
                pbc=np.concatenate([batch["pbc"]] * copies))
    shape = (len(species), n, l)
    before = tune.get_config(shape)
    tune.set_config(shape, dict(before, exp_chunk=chunk))
    try:
        al = calc.transform(rb.AtomsList(rb.StructureSet(many)), precision="fp32")
        c = al.get_features(calc, keys=calc.get_keys(sorted(species))).reshape(copies, 120, -1)
    finally:
        tune.set_config(shape, before)
    ref = O.Run(oracle_calc(rc=4.0, n=n, l=l, sigma=0.5), batch, sorted(species)).expansion().reshape(c.shape[1:])
    assert np.abs(c - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("n,l", [(1, 12), (16, 1), (11, 2), (16, 3), (13, 4), (12, 7), (16, 7), (10, 12), (16, 12)])
@pytest.mark.parametrize("chunk", [8, 16, 32])
def test_channels(n, l, chunk):
    copies_match_oracle(n, l, (8, 14), 14.0, chunk)
