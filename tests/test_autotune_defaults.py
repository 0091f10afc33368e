"""A tuning that leaves the branches out gets the untuned calculator's."""
import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import autotune as T
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.calculator import TWO_BRANCH_ATOMS, Batch, LinearModel, SO4Calculator


def test_branches_left_out_are_the_steps_own_rule():
    assert T.Choice(wkmax=4).branches == 0 and T.default_choice(8) == T.Choice()
    assert T.Choice.from_dict({"wkmax": 4, "branches": 2}).branches == 2  # a file that says two


@pytest.mark.gpu
def test_a_tuned_calculator_branches_by_the_number_of_atoms(cuda_device):
    model = None
    for cells, rule in (((5, 5, 5), 1), ((11, 11, 11), 2)):
        batch = Batch([S.diamond_si(*cells, sigma=0.05, rng=np.random.default_rng(1))])
        assert (batch.natoms > TWO_BRANCH_ATOMS) == (rule == 2)
        for tuning, want in ((None, rule), (T.Choice(wkmax=4), rule), (T.Choice(branches=1), 1), (T.Choice(branches=2), 2)):
            calc = SO4Calculator(lmax=1, rcut=3.0, kind="SNAP", weights={"Si": 1.0}, tuning=tuning)
            model = model or LinearModel(torch.linspace(-1, 1, calc.nB)[None]).cuda()
            assert calc.capture(batch, model).branches == want, (cells, tuning)
