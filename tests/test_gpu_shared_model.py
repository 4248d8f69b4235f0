"""One model on several structure sets whose species differ: its device copies
are laid out for the species of the set that used it last, so a call on another
set has to lay them out again, whatever it reuses otherwise.

Answers are compared with those of a model and a set of their own (the same
kernels: 1e-12 relative)."""
import numpy as np
import pytest

import librascal_b200 as rb
from helpers import wrap
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


def box(species, seed, n_atoms=90, side=10.0):
    rng = np.random.default_rng(seed)
    site = rng.permutation(125)[:n_atoms]
    f = (np.stack([site // 25, site // 5 % 5, site % 5], 1) + 0.5 + rng.uniform(-.2, .2, (n_atoms, 3))) / 5
    return dict(atom_offsets=np.array([0, n_atoms]), positions=f * side,
                numbers=np.resize(species, n_atoms).astype(np.int32), cells=np.array([np.eye(3) * side]),
                pbc=np.ones((1, 3), np.int32))


@pytest.fixture(scope="module")
def make_model():
    calc = soap(rc=4.0, n=6, l=4, sigma=0.4)
    batch = box([1, 8], 0)
    managers = calc.transform(rb.AtomsList(rb.StructureSet(batch)))
    keys = calc.get_keys([1, 8])
    x = managers.get_features(calc, keys=keys)
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][:30], x[:30], keys)
    return lambda: rb.GAPModel(calc, sp, np.linspace(-1, 1, 30), 2)


def close(a, b):
    return np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


def test_recorded_step_after_other_layouts(make_model):
    """FP32 on other species, then FP64 on the step's species: the FP64 copy of
    the sparse points is the step's again, the BF16 one is not."""
    a, b = box([1, 8], 1), box([1, 6, 8], 2)
    model, own = make_model(), make_model()
    st, same, other = rb.StructureSet(a), rb.StructureSet(a), rb.StructureSet(b)
    alone = rb.StructureSet(a)
    alone.use_graphs(False)
    rng = np.random.default_rng(0)
    replays = 0
    for _ in range(6):
        model.predict(other, "fp32")
        model.predict(same, "fp64")
        pos = wrap(dict(a, positions=a["positions"] + 0.02 * rng.normal(size=a["positions"].shape)))["positions"]
        before = st.md_step_info()[2]
        E, F, _ = model.md_step(st, pos)
        replays += st.md_step_info()[2] > before
        alone.update_positions(pos)
        E0, F0 = own.predict(alone, "fp32")
        assert close(E, E0) and close(F, F0)
    assert replays >= 1


@pytest.mark.parametrize("species", [[1, 6, 8], [1, 6, 7, 8], [8]])
def test_backward_after_another_forward(make_model, species):
    """Two forwards of one model, then both backwards, in either order."""
    import torch
    a, b = box([1, 8], 3), box(species, 4, n_atoms=70)
    model = make_model()
    for first in (0, 1):
        batches = [a, b]
        pos = [torch.tensor(x["positions"], device="cuda", requires_grad=True) for x in batches]
        E = [rb.gap_energy(p, model, rb.StructureSet(x)).sum() for p, x in zip(pos, batches)]
        for k in (first, 1 - first):
            (g,) = torch.autograd.grad(E[k], pos[k])
            alone = rb.StructureSet(batches[k])
            alone.use_graphs(False)
            _, F0 = make_model().predict(alone, "fp32")
            assert close(-g.cpu().numpy(), F0)
