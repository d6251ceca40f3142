"""Derivatives of a few grids (densities and fields) where their one-launch
kernel has remainders: meshes with points beyond the last 32 or 96, lines of
one to 35 points, grids with all axes, without Laplacian and with one axis
only (grad rho and lap rho, grad B, div W), against numpy sums.  Bars: 1e-13
norm-wise for FP64 sums of at most 35 terms, 1e-11 for double-float ones."""
import ctypes as C

import numpy as np
import pytest

from mocca_gb300 import MG_FP64, MG_MIXED, SLY4, RunParams, _abi
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


def _line(f, axis, sign, kind):
    n = f.shape[2 - axis]
    d = np.zeros((2, 2, n, n))
    _abi.load().mg_lagrange_matrices(n, C.c_double(0.8), 1, d[0].ctypes.data_as(_abi._D),
                                     d[1].ctypes.data_as(_abi._D))
    m = d[kind][1 if sign > 0 else 0]
    return np.moveaxis(np.moveaxis(f, 2 - axis, -1) @ m.T, -1, 2 - axis)


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n", [(1, 2, 3), (5, 7, 9), (12, 11, 10), (16, 17, 18), (24, 23, 25),
                               (35, 6, 31)])
@pytest.mark.parametrize("prec", [MG_FP64, MG_MIXED])
def test_field_derivatives(built, n, prec):
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=4, neutrons=2, protons=2,
                  coulomb_solver=0, precision=prec)
    rng = np.random.default_rng(5)
    bar = 1e-13 if prec == MG_FP64 else 1e-11
    shape = (n[2], n[1], n[0])
    g = MeshState(p, SLY4)
    psi = rng.normal(size=(4, 4) + shape)
    qn = np.array([[-1, 1, 1, 1], [-1, -1, 1, 1], [1, 1, 1, 1], [1, -1, 1, 1]], dtype=np.int32)
    g.set_spinors(psi, qn)
    g.set_occupations(np.array([2.0, 1.5, 1.0, 0.5]))
    g.DeriveAll()
    g.UpdateDensities()
    d = g.get_densities()
    for it in range(2):
        rho = d["rho"].reshape((2,) + shape)[it]
        for a in range(3):
            assert _rel(d["derrho"].reshape((2, 3) + shape)[it, a], _line(rho, a, 1, 0)) < bar
        lap = sum(_line(rho, a, 1, 1) for a in range(3))
        assert _rel(d["laprho"].reshape((2,) + shape)[it], lap) < bar
    g.ConstructPotentials()
    f = g.get_potentials()
    W = f["W"].reshape((2, 3, 3) + shape)
    # signs of W (mu, nu) along each axis: (parity, signature, component) as for
    # the preconditioner's classes
    cls = {(0, 1): (-1, 1, 1), (0, 2): (-1, -1, 2), (1, 2): (-1, -1, 1)}

    def signs(mu, nu):
        P, S, comp = cls[tuple(sorted((mu, nu)))]
        return (S if comp in (1, 4) else -S, 1 if comp in (1, 3) else -1,
                S * P if comp in (1, 2) else -S * P)

    for it in range(2):
        B = f["B"].reshape((2,) + shape)[it]
        for a in range(3):
            assert _rel(f["nablaB"].reshape((2, 3) + shape)[it, a], _line(B, a, 1, 0)) < bar
        for nu in range(3):
            parts = [_line(W[it, nu, mu], mu, signs(mu, nu)[mu], 0) for mu in range(3) if mu != nu]
            got = f["divW"].reshape((2, 3) + shape)[it, nu]
            scale = max(np.linalg.norm(q) for q in parts)
            assert np.linalg.norm(got - sum(parts)) < bar * scale
    g.close()
