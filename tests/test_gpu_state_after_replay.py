"""What a handle may reuse after a recorded MD step was replayed on it: nothing.
A replay overwrites the positions, the neighbour list, the row order and the
FP32 features, so an FP64 prediction or an autograd backward that follows must
not take what an earlier call left for them."""
import numpy as np
import pytest

import librascal_b200 as rb
from helpers import wrap
from librascal_b200 import _native as N
from test_gpu_md import setup_box

pytestmark = pytest.mark.gpu


def moved(batch, pos, rng):
    return wrap(dict(batch, positions=pos + 0.05 * rng.normal(size=pos.shape)))["positions"]


def test_fp64_between_replays():
    """FP32 MD with an FP64 check now and then, each against a fresh handle.
    Both run the same kernels; FP64 differs by the order of atomic additions
    (1e-12 relative). The positions move by 0.05 A, which changes the forces in
    the first digits."""
    batch, model = setup_box(seed=11)
    st = rb.StructureSet(batch)
    rng = np.random.default_rng(0)
    pos = batch["positions"]
    for _ in range(5):
        # the first steps record again while buffers still grow; the later ones replay
        for _ in range(2):
            pos = moved(batch, pos, rng)
            model.md_step(st, pos)
        E, F = model.predict(st, "fp64")
        E0, F0 = model.predict(rb.StructureSet(dict(batch, positions=pos)), "fp64")
        assert np.abs(E - E0).max() <= 1e-12 * np.abs(E0).max()
        assert np.abs(F - F0).max() <= 1e-12 * np.abs(F0).max()
    assert st.md_step_info()[2] >= 1  # the last steps were replays


def test_backward_after_a_replay_is_refused():
    import torch
    batch, model = setup_box(seed=12)
    st = rb.StructureSet(batch)
    pos = torch.tensor(batch["positions"], dtype=torch.float64, device="cuda")
    E = torch.empty(1, dtype=torch.float64, device="cuda")
    g = torch.ones(1, dtype=torch.float64, device="cuda")
    out = torch.empty((st.n_atoms, 3), dtype=torch.float64, device="cuda")
    rng = np.random.default_rng(1)
    steps = 0
    for _ in range(4):
        N.check(N.lib().rgpu_gap_forward_dev(model.handle, st.handle, pos.data_ptr(), E.data_ptr()))
        before = st.md_step_info()[2]
        model.md_step(st, moved(batch, batch["positions"], rng))
        steps += st.md_step_info()[2] > before
        rc = N.lib().rgpu_gap_backward_dev(model.handle, st.handle, g.data_ptr(), out.data_ptr())
        assert rc == N.ERR_NOT_COMPUTED
    assert steps >= 1  # at least one of them was a replay


def test_list_after_a_replay_is_refused():
    batch, model = setup_box(seed=13)
    st = rb.StructureSet(batch)
    for _ in range(3):
        model.md_step(st, batch["positions"])
    st.build_neighbour_list(4.0)
    before = st.md_step_info()[2]
    model.md_step(st, batch["positions"])
    assert st.md_step_info()[2] == before + 1
    with pytest.raises(RuntimeError, match="neighbour list has not been built"):
        st.neighbour_list()
