"""The neighbour list where its kernels change: one CTA or several for the bins (640 atoms,
4,096 bins), four warps or one per centre (1,216 centres), keys ranked from registers or from
memory (64 images), pairs of a centre with more than 32 images, with and without images of its
own.  Bit for bit the oracle's list: no tolerance.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyxtal_ff_gb300 import engine
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.calculator import Batch, LinearModel, SO4Calculator

pytestmark = pytest.mark.gpu


def _si(*n):
    return S.diamond_si(*n, sigma=0.1, rng=np.random.default_rng(71 + sum(n)))


CASES = {
    "640 atoms": ([_si(5, 4, 4)], 3.0),
    "648 atoms": ([_si(9, 3, 3)], 3.0),
    "1216 atoms": ([_si(19, 8, 1)], 3.0),
    "1224 atoms": ([_si(17, 9, 1)], 3.0),
    "more than 4096 bins": ([S.Atoms([14] * 5, np.random.default_rng(72).uniform(0, 90, (5, 3)), 90 * np.eye(3)),
                             _si(1, 1, 1)], 5.2),
    "64 images and more": ([_si(1, 1, 1), S.Atoms([14], [[0.1, 0.2, 0.3]], 2.8 * np.eye(3)), _si(2, 1, 1)], 6.9),
    "no periodicity": ([S.Atoms([14] * 40, np.random.default_rng(73).uniform(0, 9, (40, 3)), 9 * np.eye(3), pbc=False)],
                       4.0),
}


@pytest.mark.parametrize("case", CASES)
def test_neighbour_list_is_the_oracles(cuda_device, case):
    structs, rcut = CASES[case]
    batch = Batch(structs)
    pos = torch.from_numpy(batch.positions).cuda()
    nb = engine.build_neighbors(pos, batch.cells, batch.pbc, batch.atom_ptr, rcut)
    lay = engine.layout(batch.cells, batch.pbc, batch.atom_ptr, rcut)
    slots = int(torch.diff(nb.img_ptr).max()) + 8
    lite = engine.NeighborBuffers.allocate(lay, nb.nimg + 64, nb.npair + 64, "cuda", slot_cap=slots)
    engine.enqueue_neighbors(lay, pos, lite, lite=True, count_pairs=False)
    M, P, bits = [int(v) for v in lite.summary_dev().cpu()]
    assert M == nb.nimg and P == 0 and engine.check_summary(M, P, bits, lite.cap_m, lite.cap_p)
    for key in ("img_j", "img_off", "img_r", "img_rev"):
        assert torch.equal(getattr(lite, key)[:M], getattr(nb, key)), key
    assert torch.equal(lite.img_ptr, nb.img_ptr)
    h = {k: getattr(nb, k).cpu().numpy() for k in ("img_ptr", "pair_ptr", "img_j", "img_off", "img_r", "seq", "pair_img",
                                                    "nsite", "img_pair")}
    for s, at in enumerate(structs):
        ref = O.NeighborList(at.positions, at.get_cell(), at.get_pbc(), rcut)
        a0, a1 = batch.atom_ptr[s], batch.atom_ptr[s + 1]
        m0, m1, p0, p1 = h["img_ptr"][a0], h["img_ptr"][a1], h["pair_ptr"][a0], h["pair_ptr"][a1]
        assert np.array_equal(h["img_ptr"][a0:a1 + 1] - m0, ref.img_ptr)
        assert np.array_equal(h["img_j"][m0:m1] - a0, ref.img_j) and np.array_equal(h["img_off"][m0:m1], ref.img_off)
        assert np.array_equal(h["img_r"][m0:m1], ref.img_r) and np.array_equal(h["seq"][p0:p1], ref.seq)
        assert np.array_equal(h["pair_img"][p0:p1 + 1] - m0, ref.pair_img[: p1 - p0 + 1])
        assert np.array_equal(h["nsite"][a0:a1] - p0, ref.nsite)
        assert np.array_equal(h["img_pair"][m0:m1] - p0, np.repeat(np.arange(p1 - p0), np.diff(ref.pair_img[: p1 - p0 + 1])))


@pytest.mark.parametrize("cells,branches", [((1, 1, 1), 1), ((19, 8, 8), 1), ((17, 13, 11), 2)])
def test_captured_step_is_compute(cuda_device, cells, branches):
    """The captured step (its list in one or two branches: 8, 9,728 and 19,448 atoms) against the
    uncaptured call, bit for bit, and positions whose list outgrows the buffers (or does not:
    the 8 atoms')."""
    batch = Batch([_si(*cells)])
    calc = SO4Calculator(lmax=1, rcut=4.9, kind="SNAP", weights={"Si": 1.0})
    model = LinearModel(torch.linspace(-1, 1, calc.nB)[None]).cuda()
    step = calc.capture(batch, model)
    assert step.branches == branches
    pos = batch.positions + np.random.default_rng(74).normal(0, 0.02, batch.positions.shape)
    out, ref = step(pos), calc.compute(batch, model, positions=pos)
    assert step.check()
    for key in ("energy", "forces", "stress", "x"):
        assert torch.equal(out[key], ref[key]), key
    step(0.5 * pos)
    nb = calc.neighbors(batch, torch.from_numpy(0.5 * pos).cuda())
    assert step.check() == (nb.nimg <= step.cap_m and int(torch.diff(nb.img_ptr).max()) <= step.slot_cap)
    out = step(pos)
    assert step.check() and torch.equal(out["forces"], ref["forces"])
