"""The neighbour list and the row sorts at the sizes where their kernels
branch: batches around the one-launch scan, the one-block row sort and the
one-block structure setup, boxes with more sites than a warp, many empty boxes,
and list capacities outgrown in a recorded step.

The list is compared bit for bit with the oracle; energies and forces with the
FP64 path at the FP32 bar (1e-4 of the largest force; energies to 1e-6 of the
sum of their terms, about ten FP32 roundings each)."""
import numpy as np
import pytest

import librascal_b200 as rb
from librascal_b200 import synthetic
from oracle import oracle as O
from test_gpu_parity import oracle_calc, soap

pytestmark = pytest.mark.gpu


def grid_box(n_atoms, side, seed, species=(8, 14)):
    rng = np.random.default_rng(seed)
    g = int(np.ceil(n_atoms ** (1 / 3)))
    site = rng.permutation(g ** 3)[:n_atoms]
    f = (np.stack([site // g // g, site // g % g, site % g], 1) + 0.5 + rng.uniform(-.3, .3, (n_atoms, 3))) / g
    return dict(atom_offsets=np.array([0, n_atoms]), positions=f * side,
                numbers=rng.choice(species, n_atoms).astype(np.int32), cells=np.array([np.eye(3) * side]),
                pbc=np.ones((1, 3), np.int32))


# a crowded box (about 200 sites per bin), a cell smaller than the cutoff (125 images), and cluster batches of 511..513
# structures (one setup block or a scan of its own; about 100 000 mostly empty bins)
@pytest.mark.parametrize("case", ["crowded", "images", "clusters511", "clusters512", "clusters513"])
def test_list_matches_the_oracle(case):
    if case == "crowded":
        batch, rc = grid_box(700, 6.0, 1), 4.0
    elif case == "images":
        batch, rc = grid_box(5, 2.5, 2), 4.0
    else:
        batch, rc = synthetic.molecule_clusters(n_struct=int(case[8:]), n_min=3, n_max=5, seed=3), 4.0
    st = rb.StructureSet(batch)
    st.build_neighbour_list(rc)
    g = st.neighbour_list()
    r = O.Run(oracle_calc(rc=rc), batch, np.unique(batch["numbers"]))
    p = r.pairs()
    for key in ("j", "shift", "distance", "direction"):
        assert np.array_equal(g[key], p[key]), key


# centres around the one-block sort's 4 096 and past the one-launch scan's 8 192
@pytest.mark.parametrize("n_atoms", [31, 1025, 4095, 4096, 4097, 8193])
def test_row_sorts(n_atoms):
    batch = grid_box(n_atoms, 2.3 * n_atoms ** (1 / 3), n_atoms, species=(1, 6, 8))
    calc = soap(rc=4.0, n=4, l=2, sigma=0.4)
    st = rb.StructureSet(batch)
    managers = calc.transform(rb.AtomsList(st))
    keys = calc.get_keys([1, 6, 8])
    x = managers.get_features(calc, keys=keys)
    rng = np.random.default_rng(1)
    pick = rng.choice(n_atoms, size=30)
    alpha = rng.normal(size=30)
    sp = rb.SparsePoints(calc)
    sp.add_dense(batch["numbers"][pick], x[pick], keys)
    model = rb.GAPModel(calc, sp, alpha, 2)
    E0, F0 = model.predict(st, "fp64")
    for _ in range(2):  # the ordinary path, then its recording
        E, F = model.predict(st, "fp32")
        assert np.abs(E - E0).max() <= 1e-6 * n_atoms * np.abs(alpha).sum()
        assert np.abs(F - F0).max() <= 1e-4 * np.abs(F0).max()


def test_layouts_in_turn_on_one_handle():
    """Two models of different (n, l) on one handle: the recorded call of the
    first still finds its own column map after the second has run."""
    batch = grid_box(120, 11.0, 9)
    st = rb.StructureSet(batch)
    models, refs = [], []
    for n, l in [(6, 3), (4, 2)]:
        calc = soap(rc=4.0, n=n, l=l, sigma=0.4)
        managers = calc.transform(rb.AtomsList(rb.StructureSet(batch)))
        keys = calc.get_keys([8, 14])
        x = managers.get_features(calc, keys=keys)
        sp = rb.SparsePoints(calc)
        sp.add_dense(batch["numbers"][:20], x[:20], keys)
        models.append(rb.GAPModel(calc, sp, np.linspace(-1, 1, 20), 2))
        refs.append(models[-1].predict(rb.StructureSet(batch), "fp64")[1])
    for k in [0, 0, 1, 1, 0, 1, 0, 0, 1]:
        _, F = models[k].predict(st, "fp32")
        assert np.abs(F - refs[k]).max() <= 1e-4 * np.abs(refs[k]).max()
    for k in [0, 0, 1, 0, 0, 1, 1, 0]:
        _, F, _ = models[k].md_step(st, batch["positions"])
        assert np.abs(F - refs[k]).max() <= 1e-4 * np.abs(refs[k]).max()
