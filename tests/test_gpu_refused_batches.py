"""A batch that StructureSet.set refuses leaves the former one in place, on the
host and on the device: later calls answer for it, whatever the sizes of the
refused one were. Compared with the answers before the refusal (the same
kernels: 1e-12 relative)."""
import numpy as np
import pytest

import librascal_b200 as rb
from helpers import wrap
from test_gpu_md import setup_box

pytestmark = pytest.mark.gpu


def refused(batch, how):
    n = len(batch["numbers"])
    bad = dict(batch)
    if how == "type":
        bad["numbers"] = np.where(np.arange(n) == 3, 130, batch["numbers"]).astype(np.int32)
    elif how == "more atoms":  # fifty times the atoms, one of them of no known type
        bad = dict(atom_offsets=np.array([0, 50 * n]), positions=np.tile(batch["positions"], (50, 1)),
                   numbers=np.tile(batch["numbers"], 50), cells=batch["cells"], pbc=batch["pbc"])
        bad["numbers"][-1] = -1
    elif how == "more structures":
        bad = dict(atom_offsets=np.concatenate([np.arange(n), [n - 2]]), positions=batch["positions"],
                   numbers=batch["numbers"], cells=np.tile(batch["cells"], (n, 1, 1)), pbc=np.tile(batch["pbc"], (n, 1)))
    elif how in ("nan", "inf"):
        bad["cells"] = np.array(batch["cells"])
        bad["cells"][0, 1, 1] = float(how)
    else:
        bad["atom_offsets"] = np.array([1, n])
    return bad


@pytest.mark.parametrize("how", ["type", "more atoms", "more structures", "first offset", "nan", "inf"])
def test_former_batch_stays(how):
    batch, model = setup_box(seed=31)
    st = rb.StructureSet(batch)
    bad = refused(batch, how)
    pos = wrap(dict(batch, positions=batch["positions"] + 0.03))["positions"]
    E0, F0 = model.predict(st, "fp64")
    st.update_positions(pos)
    E1, F1 = model.predict(st, "fp64")
    steps = [model.md_step(st, pos, stress=True) for _ in range(3)]
    st.update_positions(batch["positions"])

    def close(a, b):
        return np.abs(a - b).max() <= 1e-12 * np.abs(b).max()

    with pytest.raises(RuntimeError):
        st.set(bad)
    assert (st.n_structures, st.n_atoms) == (1, len(batch["numbers"])) and st.batch["numbers"] is batch["numbers"]
    E, F = model.predict(st, "fp64")
    assert close(E, E0) and close(F, F0)
    with pytest.raises(RuntimeError):
        st.set(bad)
    st.update_positions(pos)
    E, F = model.predict(st, "fp64")
    assert close(E, E1) and close(F, F1)
    with pytest.raises(RuntimeError):
        st.set(bad)
    for a, b in zip(model.md_step(st, pos, stress=True), steps[-1]):
        assert close(a, b)
