"""How often compute() of a linear energy builds its neighbour list where the arrays' first capacity
is too small: at most twice (the second with the counts of the first), once where the structure's
density tells.  Results against a call whose arrays fitted, bit for bit."""
import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import engine
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.calculator import Batch, LinearModel, SO4Calculator


def _layout(n, vol, rcut, pbc=1):
    ptr = np.array([0, n])
    images = engine._images_by_density(ptr, [vol], np.full((1, 3), pbc), rcut)
    return engine.Layout(n, 1, ptr, np.array([vol]), None, 27, None, None, rcut, images)


def test_capacity_of_a_list_not_seen_before():
    assert engine.capacity_for(_layout(100, 2000.0, 4.011)) == (6400, 6500)
    m, p = engine.capacity_for(_layout(108, 108 * 11.8, 7.013))  # copper: 122 images an atom
    assert 108 * 122 * 1.2 < m < 108 * 122 * 1.3 and p == m + 108
    assert engine.capacity_for(_layout(10, 0.0, 4.011, pbc=0)) == (640, 650)  # no cell
    assert engine.capacity_for(_layout(100, 1.0, 4.011, pbc=0)) == (6400, 6500)


def test_capacity_after_a_list_that_did_not_fit():
    lay = _layout(50, 1e6, 4.012)
    assert engine.more_capacity(lay, 3200, 3250, 4800, 3000) == (6016, int(4850 * 1.25) + 16)
    assert engine.more_capacity(lay, 3200, 3250, 3000, 4000) == (3766, 5016)


@pytest.mark.gpu
@pytest.mark.parametrize("case,lists", [("dense cluster", 2), ("dense crystal", 1), ("grown", 2)])
def test_lists_of_a_linear_compute(cuda_device, monkeypatch, case, lists):
    rng = np.random.default_rng(95)
    rcut = 6.017
    if case == "dense crystal":
        at = S.Atoms([14] * 108, 3.6 * np.stack(np.unravel_index(np.arange(27), (3, 3, 3)), -1).repeat(4, 0)
                     + np.tile(1.8 * np.array([[0, 0, 0], [0, 1, 1], [1, 0, 1], [1, 1, 0]]), (27, 1))
                     + rng.uniform(-0.05, 0.05, (108, 3)), 10.8 * np.eye(3))
    else:  # 100 atoms within 3.4 A a side: 99 images each
        at = S.Atoms([14] * 100, 20 + rng.uniform(-1.7, 1.7, (100, 3)), 60 * np.eye(3))
    batch = Batch([at])
    calc = SO4Calculator(lmax=2, rcut=rcut, kind="SNAP", weights={"Si": 1.0})
    model = LinearModel(torch.linspace(-1, 1, calc.nB)[None]).cuda()
    lay = engine.layout(batch.cells, batch.pbc, batch.atom_ptr, rcut)
    key = (lay.natoms, lay.nbins, lay.rcut)
    engine._NL_CAPACITY.pop(key, None)
    if case == "grown":
        engine._NL_CAPACITY[key] = (8000, 8000)
    calls = []
    real = engine.enqueue_neighbors
    monkeypatch.setattr(engine, "enqueue_neighbors", lambda *a, **k: (calls.append(1), real(*a, **k))[1])
    out = calc.compute(batch, model)
    assert len(calls) == lists
    assert out["neighbors"].nimg > 64 * batch.natoms
    ref = calc.compute(batch, model)
    assert len(calls) == lists + 1  # it fits from now on
    for k in ("energy", "forces", "stress", "x"):
        assert torch.equal(out[k], ref[k]), k
