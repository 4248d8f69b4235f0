"""Recorded predictions of both kinds, energies alone and forces, in turn over
as many sizes as a handle keeps: once each is recorded, every call replays. Each
answer is compared with the ordinary path of a handle of its own (the same
kernels: 1e-12 relative)."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import synthetic
from test_gpu_graphs import _close, _model

pytestmark = pytest.mark.gpu


def first(batch, count):
    off = batch["atom_offsets"][:count + 1]
    return dict(batch, atom_offsets=off, positions=batch["positions"][:off[-1]], numbers=batch["numbers"][:off[-1]],
                cells=batch["cells"][:count], pbc=batch["pbc"][:count])


@pytest.mark.parametrize("sizes", [1, 3, 4])
def test_energies_and_forces_in_turn(sizes):
    whole = synthetic.molecule_clusters(n_struct=24, seed=41)
    model, *_ = _model(whole)
    batches = [first(whole, 24 - 2 * k) for k in range(sizes)]
    expected = []
    for b in batches:
        ordinary = rb.StructureSet(b)
        ordinary.use_graphs(False)
        expected.append(model.predict(ordinary, "fp32"))
    st = rb.StructureSet(whole)

    def turn():
        for b, (E0, F0) in zip(batches, expected):
            st.set(b)
            E, _ = model.predict(st, "fp32", forces=False)
            _, F = model.predict(st, "fp32", energies=False)
            assert _close(E, E0) and _close(F, F0)

    for _ in range(5):  # buffers grow, both kinds are recorded
        turn()
    held, replays, records, _ = st.graph_info()
    assert held == 2 * sizes
    turn()
    assert st.graph_info()[:3] == (held, replays + 2 * sizes, records)


def test_energies_once_or_twice_make_no_recording_of_their_own():
    batch = synthetic.molecule_clusters(n_struct=12, seed=42)
    model, *_ = _model(batch)
    st = rb.StructureSet(batch)
    E1, _ = model.predict(st, "fp32", forces=False)
    assert st.graph_info()[:3] == (0, 0, 0)
    model.predict(st, "fp32", energies=False)
    assert st.graph_info()[:3] == (1, 0, 1)
    E2, _ = model.predict(st, "fp32", forces=False)  # the full recording
    assert st.graph_info()[:3] == (1, 1, 1)
    E3, _ = model.predict(st, "fp32", forces=False)
    assert st.graph_info()[:3] == (2, 1, 2)
    E4, _ = model.predict(st, "fp32", forces=False)
    assert st.graph_info()[1] == 2
    assert _close(E2, E1) and _close(E3, E1) and _close(E4, E1)


def test_more_sizes_than_a_handle_keeps():
    whole = synthetic.molecule_clusters(n_struct=24, seed=43)
    model, *_ = _model(whole)
    st = rb.StructureSet(whole)
    for _ in range(3):
        for k in range(6):
            st.set(first(whole, 24 - k))
            model.predict(st, "fp32")
            model.predict(st, "fp32", forces=False)
    assert st.graph_info()[0] <= 8
