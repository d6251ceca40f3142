"""Density sums on meshes and basis sizes where their splits have remainders:
mesh points not a multiple of the reduction's 32, fewer groups than its eight
warps, and groups that do not divide evenly; FP64 and mixed, against the
oracle.  Bars: the FP64 form's 1e-12 and the mixed derivatives' 1e-11
(norm-wise); div J of the mixed form, a difference of products of two
derivatives, ten times that."""
import numpy as np
import pytest

import oracle as O
from conftest import rel
from mocca_gb300 import MG_FP64, MG_MIXED, SLY4, RunParams, synthetic
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,nwt", [(5, 6, 7, 4), (9, 11, 13, 18), (16, 10, 8, 26)])
def test_density_sums(built, nx, ny, nz, nwt):
    p = RunParams(nx=nx, ny=ny, nz=nz, dx=0.8, nwt=nwt, neutrons=4, protons=4)
    psi, qn, en = synthetic.ho_basis(p, nwt // 2 - 1, seed=3)
    occ = np.random.default_rng(4).uniform(0.0, 2.0, nwt)
    occ[nwt // 3] = 0.0
    o = O.OracleState(p, SLY4)
    g = MeshState(p, SLY4)
    for s in (g, o):
        s.set_spinors(psi, qn)
        s.set_energies(en)
        s.set_occupations(occ)
        s.DeriveAll()
        s.UpdateDensities()
    want = o.get_densities()
    got = g.get_densities()
    for k in want:
        assert rel(got[k], want[k]) < 1e-12, k
    g.set_precision(MG_MIXED)
    g.DeriveAll()
    g.UpdateDensities()
    got = g.get_densities()
    for k in want:
        assert rel(got[k], want[k]) < (1e-10 if k == "nablaj" else 1e-11), k
    g.set_precision(MG_FP64)
    g.close()
