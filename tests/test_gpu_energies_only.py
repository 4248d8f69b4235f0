"""Energies without forces skip the force half and leave the energies as they
were: bit for bit those of the full call (same kernels, same order; the
structures here have at most 29 atoms, so one warp adds all of a structure's
rows or the FP64 atomics differ by rounding), on the ordinary path and on
replays, in any order of the kinds of call."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import synthetic
from test_gpu_parity import gap_setup, soap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("graphs", [False, True])
def test_energies_alone(precision, graphs):
    batch = synthetic.molecule_clusters(n_struct=25, seed=8)
    kw = dict(rc=5.0, n=8, l=6, sigma=0.4)
    _, T, sps, alpha, species = gap_setup(batch, kw, n_sparse=7)
    calc = soap(**kw)
    sp = rb.SparsePoints(calc)
    sp.add_dense(sps, T, calc.get_keys(species))
    model = rb.GAPModel(calc, sp, alpha, 2)
    ref = rb.StructureSet(batch)
    ref.use_graphs(False)
    E0, F0 = model.predict(ref, precision)
    st = rb.StructureSet(batch)
    st.use_graphs(graphs)
    tol = 1e-13 * np.abs(E0).max()  # the order of FP64 atomics
    for kind in ["e", "e", "f", "ef", "e", "f", "ef", "e"]:
        st.invalidate()
        E, F = model.predict(st, precision, energies="e" in kind, forces="f" in kind)
        assert (E is None) == ("e" not in kind) and (F is None) == ("f" not in kind)
        if E is not None:
            assert np.abs(E - E0).max() <= tol
        if F is not None:
            assert np.abs(F - F0).max() <= 1e-12 * np.abs(F0).max()
