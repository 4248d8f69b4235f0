"""get_features selects and rearranges on the device: keys in any order, twice,
absent from the batch; power spectrum and expansion, FP64 and FP32, odd and even
max_radial. The blocks of a request are those of the full export, bit for bit,
and the full export is checked against the oracle elsewhere."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [rb.SphericalInvariants, rb.SphericalExpansion])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,l", [(3, 2), (6, 4)])
def test_selected_keys(kind, precision, n, l):
    batch = synthetic.periodic_boxes(n_struct=2, side=8.0, n_atoms=20, species=(1, 6, 8), seed=n)
    calc = kind(interaction_cutoff=3.5, cutoff_smooth_width=0.5, max_radial=n, max_angular=l,
                gaussian_sigma_type="Constant", gaussian_sigma_constant=0.4)
    al = calc.transform(rb.AtomsList(rb.StructureSet(batch)), precision=precision)
    keys = calc.get_keys([1, 6, 8])
    full = al.get_features(calc, keys=keys)
    inner = calc.inner_size()
    assert full.shape == (40, len(keys) * inner) and np.abs(full).max() > 0
    at = {tuple(k): full[:, i * inner:(i + 1) * inner] for i, k in enumerate(keys.tolist())}
    absent = [7, 8] if kind is rb.SphericalInvariants else [7, 7]
    asked = [keys[-1].tolist(), absent, keys[0].tolist(), keys[-1].tolist()]
    got = al.get_features(calc, keys=np.array(asked))
    for i, k in enumerate(asked):
        want = at.get(tuple(k), np.zeros((40, inner)))
        assert np.array_equal(got[:, i * inner:(i + 1) * inner], want)
    assert al.get_features(calc, keys=np.zeros((0, 2), int)).shape == (40, 0)


def test_fp32_prediction_keeps_no_features():
    batch = synthetic.molecule_clusters(n_struct=5, seed=1)
    calc = rb.SphericalInvariants(interaction_cutoff=3.5, cutoff_smooth_width=0.5, max_radial=3, max_angular=2,
                                  gaussian_sigma_type="Constant", gaussian_sigma_constant=0.4)
    st = rb.StructureSet(batch)
    st.use_graphs(False)
    al = calc.transform(rb.AtomsList(st))
    keys = calc.get_keys(np.unique(batch["numbers"]))
    x = al.get_features(calc, keys=keys)
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][:4], x[:4], keys)
    model = rb.GAPModel(calc, sp, np.ones(4), 2)
    st.invalidate()
    model.predict(st, "fp32")
    with pytest.raises(RuntimeError):
        al.get_features(calc, keys=keys)
