"""The FP64 tensor-core GEMM at the edges of its 64 x 64 x 16 tiles, through
the sparse-kernel entry points, against numpy in the same precision.

Tolerance: an entry is a sum of D products of magnitude |t|^2 / D on average,
so its rounding error is at most D eps |t_a| |t_b| in any summation order; the
rows have unit norm and D <= 600, which gives 1.3e-13 (times zeta)."""
import numpy as np
import pytest

import librascal_b200 as rb
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


def unit_rows(rng, m, d):
    t = rng.normal(size=(m, d))
    return t / np.linalg.norm(t, axis=1, keepdims=True)


# (n, l) with D = n^2 (l + 1) for one species: odd row lengths (27, 539; 8-byte copies) and even ones, below one
# K slice (8) and several (28 slices); M around the tile's 64 and the two-tile edge
@pytest.mark.parametrize("n,l", [(2, 1), (3, 2), (8, 6), (7, 10)])
@pytest.mark.parametrize("m", [1, 63, 64, 65, 130])
def test_kmm_tile_edges(n, l, m):
    calc = soap(rc=4.0, n=n, l=l, sigma=0.4)
    d = n * n * (l + 1)
    t = unit_rows(np.random.default_rng(m), m, d)
    sp = rb.SparsePoints(calc)
    sp.add_dense([8] * m, t, calc.get_keys([8]))
    k = rb.Kernel(calc, name="GAP", zeta=2, target_type="Structure", kernel_type="Sparse")(sp)
    assert np.abs(k - (t @ t.T) ** 2).max() < 1e-12


# centres per species around the tile edge, with species of few and of many sparse points (split K, odd leading
# dimensions, a species without sparse points)
@pytest.mark.parametrize("points", [(1, 65), (33, 0), (130, 7)])
@pytest.mark.parametrize("zeta", [1, 2])
def test_knm_rows_against_features(points, zeta):
    rng = np.random.default_rng(sum(points))
    n_atoms = 150
    g = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n_atoms]
    batch = dict(atom_offsets=np.array([0, 65, n_atoms]), positions=(g + 0.5 + rng.uniform(-.2, .2, g.shape)) * 2.0,
                 numbers=rng.choice([8, 14], n_atoms).astype(np.int32), cells=np.array([np.eye(3) * 12.0] * 2),
                 pbc=np.ones((2, 3), np.int32))
    calc = soap(rc=4.0, n=3, l=2, sigma=0.4)
    managers = calc.transform(rb.AtomsList(rb.StructureSet(batch)))
    keys = calc.get_keys([8, 14])
    x = managers.get_features(calc, keys=keys)
    species = [8] * points[0] + [14] * points[1]
    t = unit_rows(rng, len(species), x.shape[1])
    sp = rb.SparsePoints(calc)
    sp.add_dense(species, t, keys)
    expected = (x @ t.T) ** zeta * (batch["numbers"][:, None] == np.array(species)[None])
    atom = rb.Kernel(calc, name="GAP", zeta=zeta, target_type="Atom", kernel_type="Sparse")(managers, sp)
    assert np.abs(atom - expected).max() < 1e-12
    rows = rb.Kernel(calc, name="GAP", zeta=zeta, target_type="Structure", kernel_type="Sparse")(managers, sp)
    sums = np.stack([expected[:65].sum(0), expected[65:].sum(0)])
    assert np.abs(rows - sums).max() < 1e-12 * 85  # up to 85 centres per structure
