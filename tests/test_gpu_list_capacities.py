"""Recorded predictions whose neighbour list outgrows its site or box capacity
(one-eighth above the recording call's counts, plus 64), in a batch of two
structures: the centres of the second lie past the capacity once the first has
grown. The replay must notice and the call fall back to the ordinary path.

`site` of a centre counts every ghost of the structures before it, so with
40 atoms in a first cell that shrinks from 14 to 5.5 A the second structure's
centres move from site 155 to site 590 of a capacity of about 500; a first cell
that grows from 5.5 to 30 A puts the second structure's boxes at 1 728 and up of
a capacity of about 690.

The results are those of a fresh handle's ordinary path, which runs the same
kernels: only the order of FP64 atomic additions differs (1e-12 relative)."""
import numpy as np
import pytest

import librascal_b200 as rb
from test_gpu_parity import soap

pytestmark = pytest.mark.gpu


def two_boxes(sides, seed=0, n_atoms=40):
    rng = np.random.default_rng(seed)
    pos = []
    for side in sides:
        site = rng.permutation(64)[:n_atoms]
        f = np.stack([site // 16, site // 4 % 4, site % 4], 1) + 0.5 + rng.uniform(-.2, .2, (n_atoms, 3))
        pos.append(f / 4 * side)
    return dict(atom_offsets=np.array([0, n_atoms, 2 * n_atoms]), positions=np.concatenate(pos),
                numbers=np.tile([1, 8], n_atoms).astype(np.int32), cells=np.array([np.eye(3) * s for s in sides]),
                pbc=np.ones((2, 3), np.int32))


@pytest.fixture(scope="module")
def model():
    calc = soap(rc=4.0, n=6, l=4, sigma=0.4)
    batch = two_boxes((9.0, 9.0))
    managers = calc.transform(rb.AtomsList(rb.StructureSet(batch)))
    keys = calc.get_keys([1, 8])
    x = managers.get_features(calc, keys=keys)
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][:12], x[:12], keys)
    return rb.GAPModel(calc, sp, np.linspace(-1, 1, 12), 2)


def close(a, b):
    return np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


# sites outgrown by the first structure, boxes by the first, boxes by the second alone
@pytest.mark.parametrize("before,after", [((14., 10.), (5.5, 10.)), ((5.5, 10.), (30., 10.)), ((10., 5.5), (10., 30.))])
@pytest.mark.parametrize("stress", [False, True])
def test_outgrown_sites_and_boxes(model, before, after, stress):
    def call(st):
        return model.predict_stress(st, "fp32") if stress else model.predict(st, "fp32")

    st = rb.StructureSet(two_boxes(before))
    call(st)
    call(st)
    assert st.graph_info()[1:3] == (1, 1)
    batch = two_boxes(after, seed=1)
    st.set(batch)
    got = call(st)
    assert st.graph_info()[1:3] == (1, 2)  # not replayed to an end: the ordinary path, recorded again
    fresh = rb.StructureSet(batch)
    fresh.use_graphs(False)
    for a, b in zip(got, call(fresh)):
        assert close(a, b)
    again = call(st)
    assert st.graph_info()[1] == 2
    for a, b in zip(again, got):
        assert close(a, b)
