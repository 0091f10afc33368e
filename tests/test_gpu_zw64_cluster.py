"""The two-atom window pass with a cluster of CTAs per group of 64 atoms: the units are only
dealt to other CTAs, and every slot is summed by one CTA in slot order, so all outputs equal
the one-atom kernel's bit for bit (B, U_tot, forces, virial, energy, JVP).

Counts of groups on both sides of the rule p groups <= 152 - 8 (p - 1): 12 and 13 (eight CTAs
to seven), 24 and 25 (five to four), 45 and 46 (three to two), 72 and 73 (two to one), and behind
one full wave of 152 (32 and 33, 72 and 73) or of 304, up to twol 6, where from 153 groups on two
CTAs of 256 threads share an SM; the last group full or holding one atom.
"""
import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import autotune
from pyxtal_ff_gb300 import structures as S
from tests.test_gpu_zw64 import _outputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("twol,nt", [(8, 512), (8, 256), (6, 512), (3, 512)])
@pytest.mark.parametrize("groups,last", [(12, 64), (13, 1), (24, 64), (25, 1), (45, 64), (46, 1), (72, 64), (73, 1), (152, 64), (153, 1), (184, 64), (185, 1),
                                         (224, 1), (225, 64), (304, 64), (305, 1), (376, 1)])
def test_cluster_split_is_bitwise_equal(cuda_device, twol, nt, groups, last):
    n = 64 * (groups - 1) + last
    full = S.diamond_si(14, 14, 16, sigma=0.1, rng=np.random.default_rng(groups))
    structs = [S.Atoms(full.numbers[:n], full.positions[:n], full.get_cell())]
    _, ref = _outputs(structs, twol, autotune.Choice(zw_atoms=32))
    _, got = _outputs(structs, twol, autotune.Choice(zw_atoms=64, zw_threads=nt))
    for k, a in ref.items():
        assert torch.equal(a, got[k]), "%s differs (twol %d, %d threads, %d atoms)" % (k, twol, nt, n)
    assert torch.isfinite(got["fl"]).all() and got["x"].abs().sum() > 0
