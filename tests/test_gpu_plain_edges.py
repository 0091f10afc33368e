"""The plain path's kernels at the edges of their work division, against the oracle.

Every compiled twol (odd ones too), and image counts on both sides of what a pass holds: 16
(FP64 matrix tiles) and 32 (one warp of set-ups), with pairs of many images that a pass cuts in
two, a centre whose only neighbours are its own images, and a last tile of centres that is
nearly empty.  Tolerances, relative to the largest value of an array: FP64 rounds V and Z once to
61 and 59 bits and sums them as integers of 2^-52.8 of a typical sum, and the recursion adds a few
2^-53 per level, amplified about tenfold where the three sections of a component cancel:
twol x 10 x 4 x 2^-53 = 5e-14 at twol 12, so 1e-12; FP32 the same with 2^-24: 2e-4 (x: 2e-5).
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.calculator import Batch, SO4Calculator

pytestmark = pytest.mark.gpu

TOL = {"fp64": (1e-12, 1e-12), "fp32": (2e-5, 2e-4)}


def _structures():
    rng = np.random.default_rng(61)
    one = S.Atoms([14], [[0.3, 0.2, 0.1]], 2.7 * np.eye(3) + rng.uniform(-0.1, 0.1, (3, 3)))
    two = S.Atoms([14, 8], [[0.1, 0.0, 0.2], [1.3, 1.5, 1.4]], np.diag([2.9, 3.1, 3.3]))
    out = [one, two, S.nacl_cluster(angle_deg=7.0)]
    out += [S.diamond_si(*n, sigma=0.1, rng=rng) for n in ((1, 1, 1), (2, 1, 1))]
    return out


def _close(got, ref, tol):
    scale = np.abs(ref).max()
    return np.abs(got - ref).max() <= tol * (scale if scale else 1.0)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("twol", range(13))
def test_plain_path_at_every_twol_and_image_count(cuda_device, twol, precision):
    w = {"Si": 1.0, "O": 0.6, "Na": 0.9, "Cl": 1.2}
    structs = _structures()
    counts = set()
    for rcut in ((3.9, 5.3) if twol > 8 else (3.2, 4.2, 5.7)):
        batch = Batch(structs)
        calc = SO4Calculator(lmax=twol / 2, rcut=rcut, kind="SNAP", weights=w, rfac0=0.97)
        out = calc.descriptors(batch, precision=precision)
        only_x = calc.descriptors(batch, precision=precision, derivative=False)["x"]
        no_stress = calc.descriptors(batch, precision=precision, stress=False)["dxdr"]
        assert torch.equal(only_x, out["x"]) and torch.equal(no_stress, out["dxdr"])
        ptr = out["pair_ptr"].cpu().numpy()
        counts |= set(np.diff(out["neighbors"].img_ptr.cpu().numpy()).tolist())
        for s, at in enumerate(structs):
            ref = O.descriptor(at, kind="SNAP", lmax=twol / 2, rcut=rcut, weights=w, rfac0=0.97, stress=True)
            a0, a1 = batch.atom_ptr[s], batch.atom_ptr[s + 1]
            p0, p1 = ptr[a0], ptr[a1]
            assert np.array_equal(out["seq"][p0:p1].cpu().numpy(), ref["seq"])
            tx, td = TOL[precision]
            assert _close(out["x"][a0:a1].cpu().numpy(), ref["x"], tx), (rcut, s)
            assert _close(out["dxdr"][p0:p1].cpu().numpy(), ref["dxdr"], td), (rcut, s)
            assert _close(out["rdxdr"][p0:p1].cpu().numpy(), ref["rdxdr"], td), (rcut, s)
    assert min(counts) < 16 < 32 < max(counts) and any(16 < c <= 32 for c in counts)


def test_plain_path_of_several_tiles_is_repeatable(cuda_device):
    # 216 centres: the last tile of 32 holds 24; the sums of warps that run in any order give
    # the same bits
    at = S.diamond_si(3, 3, 3, sigma=0.1, rng=np.random.default_rng(62))
    calc = SO4Calculator(lmax=4, rcut=5.0, kind="SNAP", weights={"Si": 1.0}, rfac0=1.0)
    for precision in ("fp64", "fp32"):
        a, b = (calc.descriptors(Batch([at]), precision=precision) for _ in range(2))
        assert all(torch.equal(a[k], b[k]) for k in ("x", "dxdr", "rdxdr"))
    ref = O.descriptor(at, kind="SNAP", lmax=4, rcut=5.0, weights={"Si": 1.0}, rfac0=1.0, stress=True)
    out = calc.descriptors(Batch([at]))
    for key in ("x", "dxdr", "rdxdr"):
        assert _close(out[key].cpu().numpy(), ref[key], 1e-12), key


def test_non_finite_weights_reach_the_outputs(cuda_device):
    # an infinite neighbour weight: whatever the digits of it would be, dB/dr is not finite
    at = S.diamond_si(1, 1, 1, sigma=0.1, rng=np.random.default_rng(63))
    calc = SO4Calculator(lmax=2, rcut=3.0, kind="SNAP", weights={"Si": float("inf")}, rfac0=1.0)
    for precision in ("fp64", "fp32"):
        out = calc.descriptors(Batch([at]), precision=precision)
        assert not torch.isfinite(out["dxdr"]).any() and not torch.isfinite(out["x"]).any()
