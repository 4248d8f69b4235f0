"""The FP64 adjoint (dE/dc per centre, then one pass over the pairs) against
the oracle's materialised gradients, at the shapes where its kernels branch:
max_angular 0 and the largest, odd max_radial (a lone last row), max_radial
above the eight channels staged at a time (two and three passes), one species
and a species that only some centres see, a species without sparse points.

Tolerance: the bar the FP64 path has had everywhere, 1e-10 of the largest
value; both sides sum the same products in FP64."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import synthetic
from test_gpu_parity import gap_setup, soap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,l,species,zeta", [(1, 0, (8,), 1), (3, 2, (1, 8), 2), (9, 3, (1, 6, 8), 2),
                                              (17, 1, (8, 14), 3), (4, 12, (1, 8), 2), (8, 7, (1, 6, 7, 8, 9), 2)])
def test_forces_and_stress(n, l, species, zeta):
    batch = synthetic.periodic_boxes(n_struct=2, side=8.0, n_atoms=23, species=species, seed=n + l)
    kw = dict(rc=3.5, n=n, l=l, sigma=0.4)
    r, T, sps, alpha, layout = gap_setup(batch, kw, n_sparse=4, zeta=zeta)
    if len(species) == 3:  # no sparse points of one central species: its centres carry no energy
        keep = sps != species[1]
        T, sps, alpha = T[keep], sps[keep], alpha[keep]
    E0, F0, S0 = r.gap_stress(sps, T, alpha, zeta)
    calc = soap(**kw)
    sp = rb.SparsePoints(calc)
    sp.add_dense(sps, T, calc.get_keys(layout))
    E, F, S = rb.GAPModel(calc, sp, alpha, zeta).predict_stress(rb.StructureSet(batch), "fp64")
    assert np.abs(E - E0).max() <= 1e-10 * np.abs(E0).max()
    assert np.abs(F - F0).max() <= 1e-10 * np.abs(F0).max()
    assert np.abs(S - S0).max() <= 1e-10 * np.abs(S0).max()
