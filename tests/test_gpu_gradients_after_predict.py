"""An FP64 prediction leaves features whose gradients can be exported, whether
it was asked for forces or for energies alone; they are those of a calculator
that was asked for gradients, bit for bit (the same kernels on the same list)."""
import numpy as np
import pytest

import librascal_b200 as rb
from test_gpu_md import setup_box
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("forces", [False, True])
def test_export_after_prediction(forces):
    batch, _ = setup_box(seed=51)
    kw = dict(rc=4.0, n=3, l=2, sigma=0.3)
    asked = soap(grads=True, **kw)
    managers = asked.transform(rb.AtomsList(rb.StructureSet(batch)))
    expected = managers.get_features_gradient(asked)
    calc = soap(**kw)
    st = rb.StructureSet(batch)
    managers = calc.transform(rb.AtomsList(st))
    keys = managers.get_keys(calc)
    x = managers.get_features(calc, keys=keys)
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][:5], x[:5], keys)
    model = rb.GAPModel(calc, sp, np.ones(5), 2)
    model.predict(st, "fp64", forces=forces)
    assert np.array_equal(managers.get_features_gradient(calc), expected)
