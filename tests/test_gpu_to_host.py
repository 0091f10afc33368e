"""engine.to_host against Tensor.cpu(): byte for byte, over the staging buffer's edges (one piece,
two halves, a last piece of one element), strided and empty tensors, several types, another stream
and two threads at once; and compute() whose neighbour list outgrows the buffers it was launched with.
"""
import threading

import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import engine
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.calculator import Batch, LinearModel, SO4Calculator

pytestmark = pytest.mark.gpu
HALF = engine.STAGE_BYTES // 2


def _same(tensors):
    ref = [None if t is None else t.cpu().numpy() for t in tensors]
    for a, b in zip(ref, engine.to_host(*tensors)):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.dtype == b.dtype and a.shape == b.shape and np.array_equal(a, b) and b.flags.writeable


@pytest.mark.parametrize("n", [1, HALF // 8, 2 * HALF // 8, 2 * HALF // 8 + 1, 5 * HALF // 8 + 1])
def test_to_host_sizes(cuda_device, n):
    gen = torch.Generator("cuda").manual_seed(n)
    d = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    _same([d, None, (1000 * d[:7]).int(), d[:0].view(0, 3), d[: n // 6 * 6].view(-1, 6).t(), d.float() > 0.5])


def test_to_host_streams_and_threads(cuda_device):
    bad = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(4):
                try:
                    _same([torch.full((HALF // 8 * (1 + i % 3) + k,), 10.0 * k + i, dtype=torch.float64, device="cuda"),
                           torch.arange(9, device="cuda") + k])
                except BaseException as e:  # reported by the test's own thread
                    bad.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_compute_repeats_a_list_that_did_not_fit(cuda_device):
    batch = Batch([S.diamond_si(2, 2, 2, sigma=0.1, rng=np.random.default_rng(81)), S.diamond_si(1, 1, 1)])
    calc = SO4Calculator(lmax=2, rcut=4.9, kind="SNAP", weights={"Si": 1.0})
    model = LinearModel(torch.linspace(-1, 1, calc.nB)[None]).cuda()
    ref = calc.compute(batch, model)
    lay = engine.layout(batch.cells, batch.pbc, batch.atom_ptr, calc.rcut)
    for cap in ((10, 5000), (5000, 10), (ref["neighbors"].nimg, ref["neighbors"].npair)):
        engine._NL_CAPACITY[(lay.natoms, lay.nbins, lay.rcut)] = cap
        out = calc.compute(batch, model)
        for key in ("energy", "forces", "virial", "stress", "x"):
            assert torch.equal(out[key], ref[key]), key
        assert out["neighbors"].nimg == ref["neighbors"].nimg and torch.equal(out["neighbors"].seq, ref["neighbors"].seq)
    bad = torch.from_numpy(batch.positions.copy())
    bad[3, 1] = float("nan")
    with pytest.raises(ValueError):
        calc.compute(batch, model, positions=bad)
    assert torch.equal(calc.compute(batch, model)["forces"], ref["forces"])
