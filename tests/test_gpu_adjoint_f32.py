"""The FP32 pair adjoint: dE/dc rows staged in shared memory or read through
the caches, each register variant (n up to 8, 12 and 16), rows of every
remainder of 16 bytes, blocks of pairs that span fewer and more centres than
they stage at a time, against the FP64 path.

Tolerance: the FP32 path's bar of 1e-4 of the largest force (of the largest
stress)."""
import numpy as np
import pytest

import librascal_b200 as rb
from test_gpu_nl_sorts import grid_box
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


def with_loose_atoms(batch, count, side):
    """`count` atoms without neighbours, in a box of their own between two copies of the batch."""
    k = int(np.ceil(count ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count]
    loose = (g + 0.5) * (side / k)
    n0 = len(batch["numbers"])
    return dict(atom_offsets=np.array([0, n0, n0 + count, 2 * n0 + count]),
                positions=np.concatenate([batch["positions"], loose, batch["positions"]]),
                numbers=np.concatenate([batch["numbers"], np.full(count, 14), batch["numbers"]]).astype(np.int32),
                cells=np.concatenate([batch["cells"], [np.eye(3) * side], batch["cells"]]),
                pbc=np.concatenate([batch["pbc"], [[1, 1, 1]], batch["pbc"]]).astype(np.int32))


@pytest.mark.parametrize("n,l", [(1, 0), (3, 1), (4, 2), (7, 3), (8, 6), (9, 4), (12, 9), (13, 5), (16, 12)])
@pytest.mark.parametrize("side,loose", [(6.0, 0), (6.0, 300), (8.5, 0), (14.0, 0)])
def test_forces(n, l, side, loose):
    # about 145, 51 and 11 neighbours per centre
    rng = np.random.default_rng(n + l)
    batch = grid_box(120, side, n + l, species=(8, 14))
    if loose:
        batch = with_loose_atoms(batch, loose, 60.0)
    calc = soap(rc=4.0, n=n, l=l, sigma=0.5)
    st = rb.StructureSet(batch)
    keys = calc.get_keys([8, 14])
    x = calc.transform(rb.AtomsList(st)).get_features(calc, keys=keys)
    pick = rng.choice(120, size=20, replace=False)
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][pick], x[pick], keys)
    model = rb.GAPModel(calc, sp, rng.normal(size=20), 2)
    E0, F0, S0 = model.predict_stress(st, "fp64")
    E, F, S = model.predict_stress(st, "fp32")
    assert np.abs(F - F0).max() <= 1e-4 * np.abs(F0).max()
    assert np.abs(S - S0).max() <= 1e-4 * np.abs(S0).max()
