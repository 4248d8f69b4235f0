"""Training matrices by (species of i, species of j) groups against the oracle:
group row counts around the GEMM's 64-row tile, rows padded to 16 columns
(odd n^2 (l + 1)), a species without sparse points, one species alone, and a
box so small that a centre sees its own images (whose gradient stays out of
row i but enters the stress).

Tolerance: 1e-10 of the block's largest value, the bar of the FP64 path; the
projection is subtracted after the GEMM, whose terms are at most a few hundred
times the result, 1e-13 relative."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import synthetic
from test_gpu_parity import gap_setup, soap
from test_gpu_training import close, gpu_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,l,species,side,atoms,zeta,drop", [
    (3, 2, (1, 8), 8.0, 21, 1, None), (5, 4, (1, 6, 8), 8.0, 30, 2, 6), (1, 0, (8,), 6.0, 9, 3, None),
    (4, 3, (8, 14), 3.0, 4, 2, None)])
def test_gradient_rows(n, l, species, side, atoms, zeta, drop):
    batch = synthetic.periodic_boxes(n_struct=2, side=side, n_atoms=atoms, species=species, seed=3 * n + l)
    kw = dict(rc=3.5, n=n, l=l, sigma=0.4)
    r, T, sps, _, layout = gap_setup(batch, kw, n_sparse=4, zeta=zeta)
    if drop is not None:
        T, sps = T[sps != drop], sps[sps != drop]
    g = gpu_kernels(soap(**kw), batch, sps, T, layout, zeta=zeta)
    ref = r.kernel_nm_derivative(sps, T, zeta, compute_neg_stress=True)
    rows = 3 * r.n_centers
    assert close(g["KD"][:rows], ref[:rows])
    assert close(g["KD"][rows:], ref[rows:])
    assert close(g["KD0"], ref[:rows])
