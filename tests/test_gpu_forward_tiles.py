"""The forward GEMM at each of its tile widths (64, 128 and 256 columns; the
sizes below pick them in turn by gemm_forward_tile's rule, with a ragged last
tile of rows and of columns each), FP32 against the FP64 path.

Tolerance: the FP32 path's bar of 1e-4 of the largest force. Energies are sums
over one 12 A box of terms alpha k^2 <= |alpha|: 1e-6 of their total, about ten
FP32 roundings of each kernel value."""
import numpy as np
import pytest

import librascal_b200 as rb
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxes,points", [(1, 97), (6, 1100), (36, 1030)])
@pytest.mark.parametrize("zeta", [2, 3])
def test_forward_tile_widths(boxes, points, zeta):
    rng = np.random.default_rng(points)
    g = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(1, -1, 3)
    pos = (g + 0.5 + rng.uniform(-.25, .25, (boxes, 216, 3))) * 2.0
    batch = dict(atom_offsets=np.arange(boxes + 1) * 216, positions=pos.reshape(-1, 3),
                 numbers=np.where(rng.random(boxes * 216) < 0.9, 8, 14).astype(np.int32),
                 cells=np.array([np.eye(3) * 12.0] * boxes), pbc=np.ones((boxes, 3), np.int32))
    calc = soap(rc=4.0, n=4, l=3, sigma=0.4)
    st = rb.StructureSet(batch)
    managers = calc.transform(rb.AtomsList(st))
    keys = calc.get_keys([8, 14])
    x = managers.get_features(calc, keys=keys)
    pick = rng.choice(len(x), size=points, replace=points > len(x))
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][pick], x[pick], keys)
    alpha = rng.normal(size=points)
    model = rb.GAPModel(calc, sp, alpha, zeta)
    E0, F0, S0 = model.predict_stress(st, "fp64")
    E, F, S = model.predict_stress(st, "fp32")
    assert np.abs(E - E0).max() <= 1e-6 * 216 * np.abs(alpha).sum()
    assert np.abs(F - F0).max() <= 1e-4 * np.abs(F0).max()
    assert np.abs(S - S0).max() <= 1e-4 * np.abs(S0).max()
