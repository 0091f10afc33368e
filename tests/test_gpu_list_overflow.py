"""Neighbour lists that outgrow a captured step's image arrays while no atom outgrows its key
slots: atoms that gather in a cluster.  check() reports it (the step is captured again), the counts
are those of the true list, and the ASE calculator goes on.  The outputs are the uncaptured call's
bit for bit: no tolerance.
"""
import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import _lib, engine
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.ase_calculator import ForceField, PyXtalFFCalculator
from pyxtal_ff_gb300.calculator import Batch, LinearModel, SO4Calculator
from pyxtal_ff_gb300.nn import NeuralNetworkPotential

RCUT, BOX = 4.0, 160.0


def _positions(nclusters, gathered):
    """nclusters groups of 32 atoms; a gathered group lies within 3 A (31 images an atom), 20 A from
    the next one; the other groups' atoms have sites of their own 6 A apart (no image)."""
    rng = np.random.default_rng(91)
    out = []
    for k in range(nclusters):
        if k in gathered:
            out.append([3.0 + 20.0 * (k % 7), 3.0 + 20.0 * (k // 7), 3.0] + rng.uniform(0, 1.7, (32, 3)))
        else:
            out.append([3.0, 3.0, 30.0] + 6.0 * np.stack(np.unravel_index(32 * k + np.arange(32), (8, 8, 16)), -1))
    return np.concatenate(out)


def _atoms(pos):
    return S.Atoms([14] * len(pos), pos, BOX * np.eye(3))


def _nets(nB):
    torch.manual_seed(7)
    nets = {"Si": torch.nn.Sequential(torch.nn.Linear(nB, 6), torch.nn.Tanh(), torch.nn.Linear(6, 1)).double()}
    return NeuralNetworkPotential(nets, {"Si": np.stack([np.zeros(nB), np.full(nB, 3.0)], 1)})


def test_summary_of_a_list_that_does_not_fit_is_not_an_error():
    capacity, offset = 1 << _lib.SO4_ERR_CAPACITY, 1 << _lib.SO4_ERR_OFFSET
    assert engine.check_summary(100, 0, 0, 128, 128)
    assert not engine.check_summary(200, 0, capacity, 128, 128)
    assert not engine.check_summary(100, 0, capacity, 128, 128)
    with pytest.raises(_lib.SO4Error):
        engine.check_summary(100, 0, capacity | offset, 128, 128)


@pytest.mark.gpu
@pytest.mark.parametrize("late", ["first", "second", "both"])
@pytest.mark.parametrize("general,branches", [(False, 1), (False, 2), (True, 1)])
def test_images_outgrow_a_captured_step(cuda_device, general, branches, late):
    n, half = 16, set(range(4)) | set(range(8, 12))  # 512 atoms; gathered clusters in both branches
    more = {"first": range(4, 8), "second": range(12, 16), "both": range(16)}[late]
    start, end = _positions(n, half), _positions(n, half | set(more))
    batch = Batch([_atoms(start)])
    calc = SO4Calculator(lmax=2, rcut=RCUT, kind="SNAP", weights={"Si": 1.0})
    if general:
        model = _nets(calc.nB).energy_model(["Si"])
        step = calc.capture(batch, model)
    else:
        model = LinearModel(torch.linspace(-1, 1, calc.nB)[None]).cuda()
        step = calc.capture(batch, model, branches=branches)
    assert step.branches == branches
    step()
    assert step.check()
    step(end)
    nb = calc.neighbors(batch, torch.from_numpy(end).cuda())
    assert nb.nimg > step.cap_m and int(torch.diff(nb.img_ptr).max()) <= step.slot_cap
    assert not step.check()
    assert int(step.nl.summary_dev()[0]) == nb.nimg
    ref = calc.compute(batch, model, positions=start)
    out = step(start)  # and back
    assert step.check()
    for key in ("energy", "forces", "stress", "x"):
        assert torch.equal(out[key], ref[key]), key


@pytest.mark.gpu
def test_ase_calculator_outlives_an_overflow(cuda_device):
    pos = [_positions(2, {0}), _positions(2, {0}), _positions(2, {0}), _positions(2, {0, 1}), _positions(2, {0, 1})]
    desc = {"type": "SNAP", "Rc": RCUT, "cutoff": "cosine", "weights": {"Si": 1.0}, "parameters": {"lmax": 2}}
    ff = ForceField(desc, _nets(SO4Calculator(lmax=2, rcut=RCUT, kind="SNAP", weights={"Si": 1.0}).nB))
    calc, atoms = PyXtalFFCalculator(ff=ff, route="adjoint"), _atoms(pos[0])
    for k, p in enumerate(pos):
        atoms.positions = p
        calc.calculate(atoms)
        assert (calc._step is None) == (k in (0, 3))
        ref = PyXtalFFCalculator(ff=ff, route="adjoint")
        ref.calculate(atoms)
        for key in ("energies", "forces", "stress"):
            assert np.array_equal(calc.results[key], ref.results[key]), key


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(2, 2, 2), (6, 6, 5)])  # four warps and one per centre
def test_offset_beyond_the_encodable_range_is_still_an_error(cuda_device, cells):
    """Images that no key can hold are left out of the counts as well as of the keys: a count without
    its key would have the sort read what the workspace held before (here bytes 0x7f)."""
    at = S.diamond_si(*cells, sigma=0.05, rng=np.random.default_rng(92))
    batch = Batch([at])
    lay = engine.layout(batch.cells, batch.pbc, batch.atom_ptr, RCUT)
    near = engine.build_neighbors(at.positions, batch.cells, batch.pbc, batch.atom_ptr, RCUT)
    pos = at.positions.copy()
    pos[5, 0] += 600 * at.get_cell()[0, 0]
    own = int(near.img_ptr[6] - near.img_ptr[5])
    for slots in (0, 64):
        bufs = engine.NeighborBuffers.allocate(lay, 2 * near.nimg, 2 * near.npair, "cuda", slot_cap=slots)
        bufs.ws.fill_(0x7f)
        engine.enqueue_neighbors(lay, torch.from_numpy(pos).cuda(), bufs)
        M, _, bits = bufs.summary_dev().tolist()
        torch.cuda.synchronize()
        assert M == near.nimg - 2 * own  # its images, and itself as the others' image
        assert bits & (1 << _lib.SO4_ERR_OFFSET) and bits & (1 << _lib.SO4_ERR_CAPACITY)
        assert not bufs.img_ptr.any()  # emptied
    with pytest.raises(_lib.SO4Error) as err:
        engine.build_neighbors(pos, batch.cells, batch.pbc, batch.atom_ptr, RCUT)
    assert err.value.code == _lib.SO4_ERR_CAPACITY
    torch.cuda.synchronize()
