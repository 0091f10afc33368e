"""so4_plain with every size of scratch: whole, cut into passes (of whole tiles of 32 centres, the last
tile ragged), its own precision's only, a header, none.  The same bits as one pass, in both
precisions, with the integers of Z' in shared memory (twol 4, 8) and in the scratch (twol 11, 12).
What was refused stays so: FP64 at twol 12 without scratch."""
import ctypes as C

import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import _lib, engine
from pyxtal_ff_gb300 import structures as S

pytestmark = pytest.mark.gpu

HEADER, NATOMS = 256, 72  # three tiles, 8 centres in the last


def _sections(twol):
    sec = lambda l: (l + 1) // 2 * (l + 1) + (l // 2 + 1 if l % 2 == 0 else 0)  # noqa: E731
    blocks = {b for l1 in range(twol + 1) for l2 in range(l1 + 1) for l in range(l1 - l2, min(twol, l1 + l2) + 1, 2)
              if l >= l1 for b in ((l1, l2, l), (l, l2, l1), (l, l1, l2))}
    return sum(sec(b[2]) for b in blocks)


def _tile_bytes(twol, precision):
    """U_tot and Z of 32 centres, and Z's integers (FP64, above twol 10) or the half rows (FP32)."""
    nz, nu = _sections(twol), sum((l + 1) ** 2 for l in range(twol + 1))
    half = sum((l // 2 + 1) * (l + 1) for l in range(twol + 1))
    if precision == 0:
        return 512 * (nu + nz + (nz if twol > 10 else 0))
    return 256 * (nu + nz + half)


class _Call:
    def __init__(self, twol, precision):
        at = S.diamond_si(3, 3, 1, sigma=0.1, rng=np.random.default_rng(99))
        n = len(at)
        assert n == NATOMS
        self.tab, self.prm = engine.tables(twol), engine.params(twol, 3.4, 0.98, "cosine")
        self.pos = torch.from_numpy(at.positions).cuda()
        self.nb = engine.build_neighbors(self.pos, at.get_cell()[None], at.get_pbc()[None], [0, n], 3.4)
        self.w = torch.linspace(0.5, 1.5, n, dtype=torch.float64, device="cuda")
        self.precision = precision

    def __call__(self, work, nbytes):
        nb, dt, p = self.nb, (torch.float64, torch.float32)[self.precision], engine._ptr
        out = [torch.full(s, np.nan, dtype=dt, device="cuda") for s in
               ((nb.natoms, self.tab.nB), (nb.npair, self.tab.nB, 3), (nb.npair, self.tab.nB, 9))]
        rc = engine.lib().so4_plain(self.tab.handle, C.byref(self.prm), self.precision, p(nb.geom), p(nb.atom_struct),
                                    nb.natoms, p(self.pos), p(self.w), p(self.w), p(nb.img_ptr), p(nb.img_j),
                                    p(nb.img_r), p(nb.pair_ptr), p(nb.pair_img), p(nb.nsite), 1, 1, *map(p, out),
                                    p(work), nbytes, engine._stream())
        return rc, out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("twol", [0, 4, 8, 11, 12])
def test_every_scratch_gives_the_same_bits(cuda_device, twol, precision):
    call = _Call(twol, precision)
    full = engine.lib().so4_plain_workspace_size(call.tab.handle, NATOMS)
    tile = _tile_bytes(twol, precision)
    assert full == HEADER + 3 * max(_tile_bytes(twol, q) for q in (0, 1))
    rc, ref = call(torch.empty(full, dtype=torch.uint8, device="cuda"), full)
    assert rc == 0 and all(torch.isfinite(t).all() for t in ref)
    for size in (HEADER + 3 * tile, HEADER + 3 * tile - 1, HEADER + tile, HEADER + tile - 1, HEADER, 0):
        for work in ([torch.empty(size + 64, dtype=torch.uint8, device="cuda")] if size else [None]):
            if work is not None:  # nothing past the size is written
                work.fill_(0x5a)
            rc, out = call(work, size)
            if size < HEADER + tile and precision == 0 and twol == 12:
                assert rc == _lib.SO4_ERR_WORKSPACE
                continue
            assert rc == 0 and all(torch.equal(a, b) for a, b in zip(out, ref)), size
            assert work is None or bool((work[size:] == 0x5a).all())


def test_without_scratch_under_capture(cuda_device):
    call = _Call(4, 1)
    full = engine.lib().so4_plain_workspace_size(call.tab.handle, NATOMS)
    _, ref = call(torch.empty(full, dtype=torch.uint8, device="cuda"), full)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rc, out = call(None, 0)
    assert rc == 0
    for _ in range(2):
        for t in out:
            t.fill_(0)
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(out, ref))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("twol", [4, 11])
def test_scratch_at_any_address(cuda_device, twol, precision):
    """A caller may carve the scratch out of a block of its own: below twol 12 and in FP32 the call
    never asked for an alignment."""
    call = _Call(twol, precision)
    full = engine.lib().so4_plain_workspace_size(call.tab.handle, NATOMS)
    block = torch.empty(full + 64, dtype=torch.uint8, device="cuda")
    assert block.data_ptr() % 32 == 0
    _, ref = call(block, full)
    for at in (4, 8, 16, 31):
        for size in (full, HEADER + _tile_bytes(twol, precision)):
            block.fill_(0x5a)
            rc, out = call(block[at:], size)
            assert rc == 0 and all(torch.equal(a, b) for a, b in zip(out, ref)), (at, size)
            assert bool((block[:at] == 0x5a).all()) and bool((block[at + size:] == 0x5a).all())
