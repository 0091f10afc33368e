"""The plain path's virial over every volume that a cell may have.

FP32: 1 / volume is FP64's, rounded once.  Two atoms with R_j = (2, 1, 4) and R_i = 0: the row (i, j)
is fl(fl(R_j / vol) t) with t = dB/dr as returned, R_j a power of two, so it is known bit for bit (two of the volumes lie so close to a tie of FP32 that an
inverse formed in FP32 rounds the other way; the last four leave FP32's normal range).
"""
import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.calculator import Batch, SO4Calculator

pytestmark = pytest.mark.gpu

RJ = np.array([2.0, 1.0, 4.0])


def _pairs(vols):
    return [S.Atoms([14, 14], [[0, 0, 0], RJ], np.diag([v, 1.0, 1.0]), pbc=False) for v in vols]


def test_fp32_virial_takes_the_rounded_fp64_inverse_volume(cuda_device):
    rng = np.random.default_rng(97)
    vols = np.concatenate([np.exp(rng.uniform(np.log(1e-2), np.log(1e7), 20000)), [469889.13875819405, 12.883346198179845, 1e-42, 1e-38, 1e38, 1e39]])
    batch = Batch(_pairs(vols))
    calc = SO4Calculator(lmax=1, rcut=5.0, kind="SNAP", weights={"Si": 1.0})
    out = calc.descriptors(batch, precision="fp32")
    ptr = out["pair_ptr"].cpu().numpy()
    rows = ptr[0:-1:2] + 1  # pairs (i, i), (i, j) of each structure's first atom
    dx, rd = out["dxdr"].cpu().numpy()[rows], out["rdxdr"].cpu().numpy()[rows]
    assert np.abs(dx).max() > 0
    with np.errstate(over="ignore", under="ignore", divide="ignore", invalid="ignore"):
        inv = (1.0 / vols).astype(np.float32)
        want = (RJ.astype(np.float32) * inv[:, None])[:, None, :, None] * dx[:, :, None, :]
    assert np.array_equal(rd, want, equal_nan=True)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_virial_of_a_cell_without_volume(cuda_device, precision):
    # molecules: the rows of a cell of volume 1, divided by 0
    rng = np.random.default_rng(98)
    for n in (2, 9, 40):  # one image per pair, and more than a pass of 32
        pos = rng.uniform(0, 3.0, (n, 3)) * [1, 1, 0.0 if n == 2 else 1.0]  # two atoms in a plane: zeros among the rows
        calc = SO4Calculator(lmax=2, rcut=4.0, kind="SNAP", weights={"Si": 1.0})
        unit, none = (calc.descriptors(Batch([S.Atoms([14] * n, pos, c, pbc=False)]), precision=precision)
                      for c in (np.eye(3), np.zeros((3, 3))))
        assert torch.equal(unit["dxdr"], none["dxdr"])
        want = unit["rdxdr"].cpu().numpy()
        with np.errstate(divide="ignore", invalid="ignore"):
            want = want / np.zeros_like(want)
        assert np.array_equal(none["rdxdr"].cpu().numpy(), want, equal_nan=True)
