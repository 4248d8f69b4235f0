"""The FP64 tensor-core GEMM with K split into planes, which the small products
of the sparse-kernel entry points take: K that the splits do not divide, a last
slice that is not full, and a split without any slice, against numpy in the same
precision.

A few centres and sparse points make a handful of 64 x 64 tiles, so the splits
are as many as K allows, K / 64: with one species D = n^2 (l + 1), with two
three times that, in slices of 16.
  (3, 8)  D  81: no split                 2 species  243: 3 of 6, 6 and 4 slices
  (5, 4)  D 125: no split                            375: 5 of 5, 5, 5, 5 and 4
  (15, 1) D 450: 7, the last one empty               1350: 21 of 5, the last four empty

Tolerance: an entry is a sum of D products of rows of unit norm, so its rounding
error is at most D eps = 3e-13 in any order of summation, for the features'
product once more that of their own reading; 1e-12, times zeta for the powers
and times the centres of a structure for its sum."""
import numpy as np
import pytest

import librascal_b200 as rb
from test_gpu_fp64_gemm import unit_rows
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("species", [[8], [8, 14]])
@pytest.mark.parametrize("n,l", [(3, 8), (5, 4), (15, 1)])
@pytest.mark.parametrize("zeta", [1, 2])
def test_split_rows(species, n, l, zeta):
    rng = np.random.default_rng(n + l)
    n_atoms = 60
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n_atoms]
    batch = dict(atom_offsets=np.array([0, 20, n_atoms]), positions=(g + 0.5 + rng.uniform(-.2, .2, g.shape)) * 2.0,
                 numbers=rng.choice(species, n_atoms).astype(np.int32), cells=np.array([np.eye(3) * 8.0] * 2),
                 pbc=np.ones((2, 3), np.int32))
    calc = soap(rc=4.0, n=n, l=l, sigma=0.4)
    managers = calc.transform(rb.AtomsList(rb.StructureSet(batch)))
    keys = calc.get_keys(species)
    x = managers.get_features(calc, keys=keys)
    points = [species[i % len(species)] for i in range(23)]
    t = unit_rows(rng, len(points), x.shape[1])
    sp = rb.SparsePoints(calc)
    sp.add_dense(points, t, keys)
    order = np.argsort(points, kind="stable")  # the columns: sparse points grouped by species
    expected = (x @ t[order].T) ** zeta * (batch["numbers"][:, None] == np.array(points)[order][None])
    atom = rb.Kernel(calc, name="GAP", zeta=zeta, target_type="Atom", kernel_type="Sparse")(managers, sp)
    assert np.abs(atom - expected).max() < 1e-12 * zeta
    rows = rb.Kernel(calc, name="GAP", zeta=zeta, target_type="Structure", kernel_type="Sparse")(managers, sp)
    sums = np.stack([expected[:20].sum(0), expected[20:].sum(0)])
    assert np.abs(rows - sums).max() < 1e-12 * zeta * 40
    # the energies take the same planes through the pointwise kernel, the forces through the second product
    alpha = rng.normal(size=len(points))
    E, _ = rb.GAPModel(calc, sp, alpha, zeta).predict(managers.structures, "fp64")
    assert np.abs(E - sums @ alpha).max() < 1e-12 * zeta * 40 * np.abs(alpha).sum()
