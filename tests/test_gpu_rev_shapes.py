"""The per-image pass of twol 6 in its two launch shapes (256 threads, and 128 above 400,000 images):
the count of images is a capacity, so the same list is run through both, and every image is one
lane pair's in either: bit for bit equal forces and virials."""
import dataclasses

import numpy as np
import pytest
import torch

from pyxtal_ff_gb300 import engine
from pyxtal_ff_gb300 import structures as S
from tests.test_gpu_zw64 import _ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 1, 1), (3, 2, 1), (5, 5, 4)])
def test_per_image_pass_shapes_agree(cuda_device, cells):
    ctx = _ctx([S.diamond_si(*cells, sigma=0.1, rng=np.random.default_rng(91))], 6, None)
    x, utot = engine.forward32(ctx.tab, ctx.prm, ctx.nb, ctx.w_nb, ctx.w_site)
    beta = torch.linspace(-1, 1, x.numel(), device="cuda").view_as(x)
    assert ctx.nb.nimg < 400000
    few = engine.adjoint32(ctx.tab, ctx.prm, ctx.nb, ctx.w_nb, utot, beta)
    many = engine.adjoint32(ctx.tab, ctx.prm, dataclasses.replace(ctx.nb, nimg=400001), ctx.w_nb, utot, beta)
    for a, b in zip(few, many):
        assert torch.equal(a, b) and torch.isfinite(a).all() and a.abs().sum() > 0
