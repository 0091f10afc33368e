"""How far the FP64 plain path's dB/dr is from the true value, on a long-double evaluation of the
reference's formulas (64 bits of mantissa or more): no further than the oracle, which evaluates
the same formulas in FP64 with every operation rounded on its own.  Both round the image's r, psi
and Cayley-Klein parameters, whose errors are the largest, as often as each other; the 2-norm over
three structures of 16 and 12 atoms with about 30 images each.
"""
from fractions import Fraction
from math import factorial

import numpy as np
import pytest

from oracle import oracle as O
from pyxtal_ff_gb300 import structures as S
from pyxtal_ff_gb300.calculator import Batch, SO4Calculator

LD, CLD = np.longdouble, np.clongdouble
PI = LD("3.14159265358979323846264338327950288")
W, RFAC, RCUT = {"Si": 1.0, "O": 0.6}, 0.97, 4.9


def _ratio(f):
    return LD(str(f.numerator)) / LD(str(f.denominator))


def _cg(l1, l2, l):
    """Clebsch-Gordan coefficients of doubled indices (Racah's sum, exact up to the root)."""
    out, fa = np.zeros((l1 + 1, l2 + 1), LD), factorial
    tri = Fraction(fa((l1 + l2 - l) // 2) * fa((l1 - l2 + l) // 2) * fa((l2 - l1 + l) // 2), fa((l1 + l2 + l) // 2 + 1))
    for m1 in range(l1 + 1):
        for m2 in range(l2 + 1):
            m = m1 + m2 - (l1 + l2 - l) // 2
            if not 0 <= m <= l:
                continue
            s = Fraction(0)
            for z in range((l1 + l2 - l) // 2 + 1):
                den = [z, (l1 + l2 - l) // 2 - z, l1 - m1 - z, m2 - z, (l - l2 - l1) // 2 + m1 + z,
                       (l - l1 + l2) // 2 - m2 + z]
                if min(den) >= 0:
                    s += Fraction((-1) ** z, int(np.prod([fa(q) for q in den], dtype=object)))
            sq = tri * fa(m1) * fa(l1 - m1) * fa(m2) * fa(l2 - m2) * fa(m) * fa(l - m) * (l + 1)
            out[m1, m2] = _ratio(s) * np.sqrt(_ratio(sq))
    return out


def _wigner(a, b, da, db, twol):
    """U_l and dU_l/dr of images with conj(a) = a, conj(b) = b, full levels."""
    us, ds = [np.ones((len(a), 1, 1), CLD)], [np.zeros((3, len(a), 1, 1), CLD)]
    for l in range(1, twol + 1):
        u, d = np.zeros((len(a), l + 1, l + 1), CLD), np.zeros((3, len(a), l + 1, l + 1), CLD)
        for mb in range(l // 2 + 1):
            p, dp = us[-1][:, mb], ds[-1][:, :, mb]
            for ma in range(l):
                f, g = np.sqrt(LD(l - ma) / LD(l - mb)), np.sqrt(LD(ma + 1) / LD(l - mb))
                u[:, mb, ma] += f * a * p[:, ma]
                d[:, :, mb, ma] += f * (da * p[:, ma] + a * dp[:, :, ma])
                u[:, mb, ma + 1] -= g * b * p[:, ma]
                d[:, :, mb, ma + 1] -= g * (db * p[:, ma] + b * dp[:, :, ma])
        for mb in range(l // 2 + 1, l + 1):
            for ma in range(l + 1):
                u[:, mb, ma] = (-1) ** (mb + ma) * np.conj(u[:, l - mb, l - ma])
                d[:, :, mb, ma] = (-1) ** (mb + ma) * np.conj(d[:, :, l - mb, l - ma])
        us.append(u)
        ds.append(d)
    return us, ds


def _dxdr(at, twol):
    """dB/dr per pair in long double (SNAP weights, cosine cutoff)."""
    nl = O.NeighborList(at.positions, at.get_cell(), at.get_pbc(), RCUT)
    n, r3, rc = len(at), nl.img_r.astype(LD), LD(RCUT)
    centre = np.repeat(np.arange(n), np.diff(nl.img_ptr))
    r = np.sqrt((r3 * r3).sum(1))
    fac, e = LD(RFAC) * PI / rc, r3 / r[:, None]
    sn, cs = np.sin(fac * r), np.cos(fac * r)
    g, (x, y, z) = sn / r, r3.T
    dg, eye = ((cs * fac * r - sn) / (r * r))[None] * e.T, np.eye(3, dtype=LD)
    us, ds = _wigner(cs + 1j * g * z, g * y + 1j * g * x, -sn * fac * e.T + 1j * (dg * z + eye[2][:, None] * g),
                     dg * y + eye[1][:, None] * g + 1j * (dg * x + eye[0][:, None] * g), twol)
    w = np.array([W[s] for s in at.symbols], LD)[nl.img_j]
    f, df = LD(0.5) * (np.cos(PI * r / rc) + 1), -LD(0.5) * PI / rc * np.sin(PI * r / rc)
    tot, dus = [], []
    for l in range(twol + 1):
        t = np.zeros((n, l + 1, l + 1), CLD) + np.eye(l + 1)
        np.add.at(t, centre, (w * f)[:, None, None] * us[l])
        tot.append(t)
        dus.append(w[:, None, None] * (f[:, None, None] * ds[l] + df[:, None, None] * e.T[:, :, None, None] * us[l]))
    zs = {}

    def block(l1, l2, l):
        if (l1, l2, l) not in zs:
            c, d, out = _cg(l1, l2, l), (l1 + l2 - l) // 2, np.zeros((n, l + 1, l + 1), CLD)
            inner = np.zeros((n, l1 + 1, l2 + 1, l + 1), CLD)  # the sums over columns, per pair of rows
            terms = [(m1, m2, m1 + m2 - d) for m1 in range(l1 + 1) for m2 in range(l2 + 1) if 0 <= m1 + m2 - d <= l]
            for m1, m2, m in terms:
                inner[:, :, :, m] += c[m1, m2] * tot[l1][:, :, None, m1] * tot[l2][:, None, :, m2]
            for m1, m2, m in terms:
                out[:, m] += c[m1, m2] * inner[:, m1, m2]
            zs[l1, l2, l] = out
        return zs[l1, l2, l]

    comps = [(l1, l2, l) for l1 in range(twol + 1) for l2 in range(l1 + 1)
             for l in range(l1 - l2, min(twol, l1 + l2) + 1, 2) if l >= l1]
    t = np.zeros((len(r), len(comps), 3), LD)
    for k, (l1, l2, l) in enumerate(comps):
        for lam, zb, fac in ((l, (l1, l2, l), LD(1)), (l1, (l, l2, l1), LD(l + 1) / LD(l1 + 1)),
                             (l2, (l, l1, l2), LD(l + 1) / LD(l2 + 1))):
            t[:, k] += fac * (np.conj(dus[lam]) * block(*zb)[centre]).real.sum((2, 3)).T
    out = np.zeros((len(nl.seq), len(comps), 3), LD)
    np.add.at(out, np.repeat(np.arange(len(out)), np.diff(nl.pair_img[: len(out) + 1])), t)
    for i in range(n):
        out[nl.nsite[i]] = 0
        out[nl.nsite[i]] = -out[nl.seq[:, 0] == i].sum(0)
    return out


def _structures():
    out = [S.diamond_si(2, 1, 1, sigma=0.1, rng=np.random.default_rng(500 + k)) for k in (0, 2)]
    return out + [S.sio2_random(n_si=4, seed=1)]


def _off(got, ref):
    d = got.astype(LD) - ref
    return float((d * d).sum() / (ref * ref).sum())


def _oracle(at, twol):
    return O.descriptor(at, kind="SNAP", lmax=twol / 2, rcut=RCUT, weights=W, rfac0=RFAC)["dxdr"]


def test_long_double_evaluation_is_the_oracles_function():
    at = _structures()[2]
    for twol in (1, 4):
        assert _off(_oracle(at, twol), _dxdr(at, twol)) < (5e-15) ** 2  # 12 levels' roundings: the set-up's rounding, l times at level l


@pytest.mark.gpu
@pytest.mark.parametrize("twol", [4, 8, 12])
def test_fp64_derivative_is_no_further_off_than_fp64_by_the_formulas(cuda_device, twol):
    structs = _structures()
    batch = Batch(structs)
    calc = SO4Calculator(lmax=twol / 2, rcut=RCUT, kind="SNAP", weights=W, rfac0=RFAC)
    out = calc.descriptors(batch)
    ptr = out["pair_ptr"].cpu().numpy()
    mine, oracle = [], []
    for s, at in enumerate(structs):
        ref = _dxdr(at, twol)
        p0, p1 = ptr[batch.atom_ptr[s]], ptr[batch.atom_ptr[s + 1]]
        mine.append(_off(out["dxdr"][p0:p1].cpu().numpy(), ref))
        oracle.append(_off(_oracle(at, twol), ref))
    assert np.mean(mine) <= np.mean(oracle)
