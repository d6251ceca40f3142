"""The Coulomb multigrid (CoulombSolver = 2) on boxes whose levels end inside a
tile of 8^3 cells, are solved by one block from the finest level on, or differ
from axis to axis: the residual |b - L phi| / |b| of the 4th-order operator
reaches the tolerance asked for, in as many iterations as any box needs, and the
potential is the direct solve's within the same 1e-8 as on the cubes."""
import numpy as np
import pytest

from conftest import rel
from mocca_gb300 import MG_FP64, MG_MIXED, SLY4, RunParams, synthetic
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


def _state(n, solver, precision):
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=2, neutrons=40, protons=40,
                  precision=precision, coulomb_solver=solver, coulomb_prec=1e-10)
    x, y, z = synthetic.mesh_axes(p)
    X, Y, Z = np.meshgrid(x, y, z, indexing="ij")
    rp = np.exp(-(X ** 2 + Y ** 2) / 9.0 - Z ** 2 / (9.0 * 1.69)).transpose(2, 1, 0)
    rp *= 40.0 / (rp.sum() * p.dv)
    g = MeshState(p, SLY4)
    g.set_densities(rho=np.concatenate([rp.reshape(-1), rp.reshape(-1)]))
    g.CalculateAllMoments()
    return g


@pytest.mark.parametrize("n", [(16, 16, 16), (15, 13, 11), (18, 18, 18), (20, 20, 20),
                               (12, 44, 28), (24, 32, 40), (30, 26, 22), (52, 20, 36)])
def test_box(built, n):
    mg = _state(n, 2, MG_FP64)
    it = mg.SolveCoulomb()
    assert it <= 40, it
    assert mg.CoulombResidual() <= 1e-10
    # a second solve starts from its own solution and a clean state
    again = mg.SolveCoulomb()
    assert again <= it and mg.CoulombResidual() <= 1e-10
    direct = _state(n, 1, MG_MIXED)
    direct.SolveCoulomb()
    cm, cd = mg.get_potentials()["coulomb"], direct.get_potentials()["coulomb"]
    assert rel(cm, cd) <= 1e-8, rel(cm, cd)
    mg.close()
    direct.close()
