"""A model or calculator that is destroyed and replaced by another one of the
same size, on one structure set: the new object may lie at the old one's
address, and its device buffers at the old ones' addresses. What the set keeps
of the old one (features, recorded predictions and steps) must not answer for
the new one. Every answer is compared with a fresh structure set's ordinary
path (the same kernels: 1e-12 relative)."""
import numpy as np
import pytest

import librascal_b200 as rb
from test_gpu_md import setup_box
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


def close(a, b):
    return np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


def points(calc, batch, counts):
    """Sparse points taken from the atoms: counts[species] of each."""
    managers = calc.transform(rb.AtomsList(rb.StructureSet(batch)))
    species = sorted(counts)
    keys = calc.get_keys(species)
    x = managers.get_features(calc, keys=keys)
    pick = np.concatenate([np.flatnonzero(batch["numbers"] == z)[:counts[z]] for z in species])
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][pick], x[pick], keys)
    return sp


@pytest.mark.parametrize("call", ["predict", "md_step"])
def test_models_one_after_the_other(call):
    """A scan of zeta and of the split of 24 sparse points over the species."""
    batch, _ = setup_box(seed=21)
    species = [int(z) for z in np.unique(batch["numbers"])]
    calc = soap(rc=4.0, n=6, l=4, sigma=0.3)
    st, ordinary = rb.StructureSet(batch), rb.StructureSet(batch)
    ordinary.use_graphs(False)
    alpha = np.linspace(-1, 1, 24)
    for zeta, first in [(2, 12), (1, 12), (3, 12), (2, 8), (2, 16), (2, 12)]:
        rest = [24 - first] if len(species) == 2 else [(24 - first) // (len(species) - 1)] * (len(species) - 1)
        sp = points(calc, batch, dict(zip(species, [first] + rest)))
        model = rb.GAPModel(calc, sp, alpha[:sp.size()], zeta)
        ordinary.invalidate()
        E0, F0 = model.predict(ordinary, "fp32")
        for _ in range(3):  # the last ones replay
            E, F = model.predict(st, "fp32") if call == "predict" else model.md_step(st, batch["positions"])[:2]
            assert close(E, E0) and close(F, F0), (zeta, first)
        del model, sp


def test_calculators_one_after_the_other():
    batch, _ = setup_box(seed=22)
    st = rb.StructureSet(batch)
    for sigma in (0.3, 0.5, 0.4, 0.6):
        calc = soap(rc=4.0, n=6, l=4, sigma=sigma)
        x = calc.transform(rb.AtomsList(st)).get_features(calc)
        x0 = calc.transform(rb.AtomsList(rb.StructureSet(batch))).get_features(calc)
        assert np.array_equal(x, x0), sigma
        del calc
