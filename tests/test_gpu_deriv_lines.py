"""Derivatives of a basis at the line lengths where the tensor-core form
changes its tiles (16, 32 and 48 points), against sums in extended precision,
and of lines that have no digits (infinities, NaN, values near the ends of
the exponent range) against plain FP64 sums.

Bars (norm-wise), FP64 form: a first derivative is rounded once (1.1e-16), its
operands to 62 bits (2^-61 of a line's largest, times sqrt(32) terms, times up
to 100 of cancellation: 2.4e-16), so 4e-16; the Laplacian adds three of them
(two more roundings, sums up to three times the result): 2e-15.  Mixed form:
the 1e-11 of its 47-bit operands."""
import ctypes as C

import numpy as np
import pytest

from mocca_gb300 import MG_FP64, MG_MIXED, SLY4, RunParams, _abi, synthetic
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


def _matrices(n, folded):
    d1, d2 = np.zeros((2, n, n)), np.zeros((2, n, n))
    st = _abi.load().mg_lagrange_matrices(n, C.c_double(0.8), int(folded),
                                          d1.ctypes.data_as(_abi._D), d2.ctypes.data_as(_abi._D))
    assert st == 0
    return d1, d2


def _slot(d, qn, comp):
    P, S, TS = qn[1:]
    s = (S * TS * (1 if comp in (0, 3) else -1), TS * (1 if comp in (0, 2) else -1),
         S * P * (1 if comp in (0, 1) else -1))[d]
    return 1 if s > 0 else 0


def _reference(psi, qn, folded, dtype):
    nwt, _, nz, ny, nx = psi.shape
    mats = [_matrices(n, folded) for n in (nx, ny, nz)]
    x = psi.astype(dtype)
    der = np.zeros((nwt, 3, 4, nz, ny, nx), dtype=dtype)
    lap = np.zeros((nwt, 4, nz, ny, nx), dtype=dtype)
    with np.errstate(invalid="ignore"):
        for i in range(nwt):
            for l in range(4):
                for d in range(3):
                    s = _slot(d, qn[i], l)
                    f = np.moveaxis(x[i, l], 2 - d, -1)
                    a, b = (np.einsum("...q,iq->...i", f, m[s].astype(dtype)) for m in mats[d])
                    der[i, d, l] = np.moveaxis(a, -1, 2 - d)
                    lap[i, l] = lap[i, l] + np.moveaxis(b, -1, 2 - d)
    return der, lap


def _rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def _params(nx, ny, nz, nwt, full, precision=MG_FP64):
    sym = 0 if full else 1
    return RunParams(nx=nx, ny=ny, nz=nz, dx=0.8, pc=sym, sc=sym, tsc=sym, nwt=nwt, neutrons=8,
                     protons=8, coulomb_solver=0, precision=precision)


@pytest.mark.parametrize("nx,ny,nz,nwt,full", [
    (15, 16, 17, 10, False), (16, 5, 3, 6, False), (31, 32, 30, 2, False),
    (32, 17, 16, 8, False), (33, 12, 18, 2, False), (40, 9, 47, 2, False), (48, 34, 4, 2, False),
    (49, 6, 8, 2, False), (17, 32, 16, 6, True), (14, 13, 12, 10, True)])
def test_line_lengths(built, nx, ny, nz, nwt, full):
    p = _params(nx, ny, nz, nwt, full)
    if full:
        psi = synthetic.gaussian_hermite_spinors(p, nwt, seed=5)
        qn = np.zeros((nwt, 4), dtype=np.int32)
        qn[:, 0] = np.where(np.arange(nwt) % 2, 1, -1)
    else:
        psi, qn, _ = synthetic.ho_basis(p, nwt // 2, seed=6)
    der, lap = _reference(psi, qn, not full, np.longdouble)
    g = MeshState(p, SLY4)
    g.set_spinors(psi, qn)
    for prec, bar, bar_lap in ((MG_FP64, 4e-16, 2e-15), (MG_MIXED, 1e-11, 1e-11)):
        if prec == MG_FP64 and (max(nx, ny, nz) > 32 or 4 * nwt * nx * ny * nz * (nx + ny + nz) < 3e6):
            bar, bar_lap = 1e-15, 4e-15   # the FMA chain (longer lines, small bases)
        g.set_precision(prec)
        g.DeriveBasis()
        g.synchronize()
        d, l = g.get_derivatives()
        assert _rel(d, der) < bar, prec
        assert _rel(l, lap) < bar_lap, prec
    g.set_precision(MG_FP64)
    g.close()


@pytest.mark.parametrize("n,nwt", [(10, 30), (24, 2)])
def test_lines_without_digits(built, n, nwt):
    """One line with a NaN, one with an infinity: their outputs, and only
    theirs, are what the plain sums give (NaN and infinities in the same
    places); lines scaled to 1e-290 and 1e295 keep their relative accuracy;
    a zero line stays zero."""
    p = _params(n, n, n, nwt, False)
    psi, qn, _ = synthetic.ho_basis(p, nwt // 2, seed=8)
    psi[0, 0, 1, 2, :] *= 1e-290
    psi[0, 1, :, :, 3] = 0.0
    psi[1, 2] *= 1e295
    psi[0, 2, 4, 5, 6] = np.nan
    psi[1, 0, 3, 3, 3] = np.inf
    der, lap = _reference(psi, qn, True, np.float64)
    g = MeshState(p, SLY4)
    g.set_spinors(psi, qn)
    g.DeriveBasis()
    g.synchronize()
    d, l = g.get_derivatives()
    for got, want in ((d, der), (l, lap)):
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.array_equal(np.isinf(got), np.isinf(want))
    for i in range(2):
        for c in range(4):
            for got, want in ((d[i, 0, c], der[i, 0, c]), (d[i, 2, c], der[i, 2, c])):
                fine = np.isfinite(want)
                scale = np.abs(want[fine]).max()
                if scale > 0:
                    assert np.abs(got[fine] / scale - want[fine] / scale).max() < 1e-13
    row, ref = d[0, 0, 0, 1, 2], der[0, 0, 0, 1, 2]
    assert np.abs(row - ref).max() < 1e-13 * np.abs(ref).max()
    assert np.array_equal(d[0, 1, 1, :, :, 3], np.zeros((n, n)))
    g.set_precision(MG_MIXED)
    g.DeriveBasis()
    g.synchronize()
    d, _ = g.get_derivatives()
    assert np.isnan(d[0, 0, 2, 4, 5, :]).all()          # the NaN's x line
    assert not np.isfinite(d[1, 2, 0, :, 3, 3]).any()   # the infinity's z line
    g.set_precision(MG_FP64)
    g.close()
